"""The sphering at the channel counts where its plans change (column blocks and CTAs of
the eigensolver, splits of the covariance and of the application), and on a
covariance that is not numerically positive definite, which the Cholesky-based
eigensolver leaves to the two-sided Jacobi forms (one SM up to 128 channels, the
whole GPU above)."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _sphere(x):
    from cudamica_b200.engine import Amica
    T, n = x.shape
    with Amica(n, T, 1, 1) as e:
        e.load_data(x)
        e.preprocess()
        return e.sphere()


def _cov(x):
    xd = x.astype(np.float64)
    xc = xd - xd.mean(0)
    return xc.T @ xc / len(x)


@pytest.mark.parametrize("n", [161, 176, 192, 193, 200, 208, 209, 224, 225, 240])
def test_sphering_matches_numpy(n):
    """cond(C) <= 1e4: 1e-10 of the norm of S is 50 times eps * cond."""
    rng = np.random.default_rng(n)
    x = (rng.laplace(size=(20 * n + 50, n)) @ synth.mixing_matrix(rng, n, 50.0).T + 3.0).astype(np.float32)
    S, _, ldetS = _sphere(x)
    d, V = np.linalg.eigh(_cov(x))
    want = (V * (2.0 / np.sqrt(d))) @ V.T
    assert np.linalg.norm(S - want) < 1e-10 * np.linalg.norm(want)
    assert abs(ldetS + np.log(2.0 / np.sqrt(d)).sum()) < 1e-9


@pytest.mark.parametrize("n", [64, 100, 128, 129, 200, 256])
@pytest.mark.parametrize("pair", [(0, 1), (3, -1)])
def test_nearly_singular_covariance(n, pair):
    """Two channels that differ by a few 1e-8 of themselves: the later one's pivot lies
    below n eps max diag C.  S then carries errors of n eps |S|, and C S S C = 4 C holds to
    a few of those times |C|^(3/2): n eps sqrt(cond C) |C|."""
    rng = np.random.default_rng(n + 7)
    T = 20_000
    x = rng.laplace(size=(T, n))
    i, j = pair
    x[:, j] = x[:, i] + np.sqrt(0.8 * n * EPS * 2.0) * rng.standard_normal(T)    # var(laplace) = 2
    x = x.astype(np.float32)
    C = _cov(x)
    r = x[:, j].astype(np.float64) - x[:, i]
    assert 0.5 < r.var() / (n * EPS * np.diag(C).max()) < 0.95    # the pivot is var(x_j | the others), below this
    S, _, ldetS = _sphere(x)
    assert np.isfinite(S).all() and np.isfinite(ldetS)
    assert np.linalg.norm(S - S.T) < 1e-12 * np.linalg.norm(S)
    size, cond = np.linalg.norm(C, 2), np.linalg.cond(S) ** 2
    assert 1e12 < cond
    assert np.linalg.norm(C @ S @ S @ C - 4.0 * C, 2) < 4 * n * EPS * np.sqrt(cond) * size
