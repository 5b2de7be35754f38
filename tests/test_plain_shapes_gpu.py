"""The plain FP32 E-step at the edges of its channel layouts (32, 64, 96 and 128
lanes, channel blocks above 128) and tiles (partial, one, odd and even counts),
against the FP64 oracle on the FP32 data.  Tolerances as in the other checks of
this form (test_parity_headline_gpu.py): the LL to 2e-6 nats per sample and
channel, the sums to 2e-5 of their largest entries."""
import numpy as np
import pytest

from oracle import oracle as O
from test_parity_headline_gpu import _as_stored, _errs
from test_tile_shapes_gpu import _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,T,M,m", [(3, 4097, 2, 1), (32, 20_000, 1, 3), (33, 9_999, 2, 2), (64, 12_345, 3, 3),
                                     (65, 10_001, 2, 5), (71, 20_003, 2, 3), (96, 9_985, 1, 4), (97, 9_985, 2, 3),
                                     (128, 19_007, 1, 5), (130, 9_001, 2, 2)])
def test_plain_estep_matches_the_oracle(n, T, M, m):
    from cudamica_b200.engine import Amica
    xs, means, S, ldetS, A0, c0 = _data(n, T, M, m)
    orc = O.Oracle(_as_stored(xs, 0), M, m, A0, c0, ldetS, nthreads=8)
    orc.prepare()
    want = orc.estep()
    with Amica(n, T, M, m, precision=0) as eng:
        assert eng.kernel == "plain_fp32"
        eng.set_sphered(xs, means, S, ldetS)
        eng.init(A0, c0)
        s = eng.estep_stats()
    assert abs(s[0] - want[0]) / (n * T) < 2e-6
    errs = _errs(s, want, n, M, m)
    for k in ("vs", "s2", "us", "kn", "ln", "bd", "rn", "phi"):
        assert errs[k] < 2e-5, (k, errs[k])
