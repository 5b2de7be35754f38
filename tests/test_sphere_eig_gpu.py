"""The sphering's eigendecomposition at the edges of its split over a cluster
(1 to 8 CTAs, 1 to 16 columns per block, odd blocks, padded columns) against
numpy in FP64.  S = 2 C^(-1/2) is computed from the covariance to a few eps
times its condition number; the data here have cond(C) <= 1e4, so 1e-10 of S's
norm is 50 times eps * cond."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 32, 33, 63, 64, 65, 97, 127, 128, 129, 160, 241, 256])
def test_sphering_matches_numpy(n):
    from cudamica_b200.engine import Amica
    rng = np.random.default_rng(n)
    T = 20 * n + 50
    x = (rng.laplace(size=(T, n)) @ synth.mixing_matrix(rng, n, 50.0).T + 3.0).astype(np.float32)
    with Amica(n, T, 1, 1) as eng:
        eng.load_data(x)
        eng.preprocess()
        S, mean, ldetS = eng.sphere()
    xd = x.astype(np.float64)
    xc = xd - xd.mean(0)
    d, V = np.linalg.eigh(xc.T @ xc / T)
    want = (V * (2.0 / np.sqrt(d))) @ V.T
    assert np.allclose(mean, xd.mean(0), rtol=1e-12, atol=1e-13)
    assert np.linalg.norm(S - want) < 1e-10 * np.linalg.norm(want)
    assert abs(ldetS + np.log(2.0 / np.sqrt(d)).sum()) < 1e-9

