"""The plain E-step's persistent grid holds every CTA that the registers allow: two
per SM for one mixture of up to 32 channels (whose time halves with it), one above."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,M,m,per_sm", [(2, 1, 1, 2), (32, 1, 1, 2), (16, 2, 1, 2), (33, 1, 1, 1), (32, 1, 5, 1)])
def test_clusters_that_fit(n, M, m, per_sm):
    import torch
    from cudamica_b200.engine import Amica
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    with Amica(n, 64 * 2 * sms, M, m, precision=0) as e:
        assert e.kernel == "plain_fp32"
        # clusters of two CTAs may leave an SM over where a unit has an odd number
        assert e.set_grid(0) >= (per_sm * sms) // M * (0.9 if M > 1 else 1.0)
