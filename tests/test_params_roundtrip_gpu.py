"""Parameters in and out of a context: any subset of them, through the staged
copy (small contexts) and past its size limit (2 MiB; n = 256, M = 4 holds 4 MiB).
Exact: nothing is computed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("A", "c", "gm", "alpha", "mu", "beta", "rho")


@pytest.mark.parametrize("n,M,m", [(2, 1, 1), (33, 2, 3), (256, 4, 5)])
@pytest.mark.parametrize("subset", [KEYS, ("A", "gm"), ("mu",), ("c", "alpha", "rho"), ("gm",), ()])
def test_params_roundtrip(n, M, m, subset):
    from cudamica_b200.engine import Amica
    rng = np.random.default_rng(n + len(subset))
    with Amica(n, 64, M, m) as eng:
        eng.init()
        before = eng.params()
        new = {k: rng.standard_normal(before[k].shape) for k in subset}
        given = {k: v.copy() for k, v in new.items()}
        eng.set_params(**given)
        for v in given.values():
            v.fill(np.nan)                    # the caller's arrays have been read
        after = eng.params()
        for k in KEYS:
            assert np.array_equal(after[k], new.get(k, before[k])), k
