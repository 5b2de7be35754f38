"""W = A^{-1} above 128 channels, whose columns are spread over a cluster in panels
of 16: one and several panels a CTA, a last panel of 1 to 16 columns, row groups
of 32 that are partly padding, pivots far from the diagonal, and a zero column
(no pivot) in the first, a middle and the last panel.

Elimination with partial pivoting leaves a residual W A - I of a modest multiple
of n eps cond(A); cond(A) = 50 and n <= 256, so 64 n eps cond(A) is 1.8e-10."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu


def _engine(n, M):
    from cudamica_b200.engine import Amica
    T = 4 * n
    eng = Amica(n, T, M, 1)
    rng = np.random.default_rng(n)
    eng.set_sphered(rng.standard_normal((T, n)).astype(np.float32))
    eng.init()
    return eng, rng


@pytest.mark.parametrize("n,M", [(129, 1), (143, 2), (144, 1), (145, 1), (160, 3), (193, 1), (241, 1),
                                 (255, 2), (256, 4)])
def test_inverse_matches_numpy(n, M):
    eng, rng = _engine(n, M)
    with eng:
        A = np.stack([synth.mixing_matrix(rng, n, 50.0)[rng.permutation(n)] for _ in range(M)])
        eng.set_params(A=A)                 # column-major per model: A[h] is A_h transposed
        eng.estep_stats()
        W = eng.params()["W"]
    for h in range(M):
        res = W[h].T @ A[h].T - np.eye(n)
        assert np.abs(res).max() < 64 * n * np.finfo(np.float64).eps * 50.0


@pytest.mark.parametrize("n,col", [(129, 0), (129, 128), (160, 100), (256, 255)])
def test_singular_matrix_is_an_error(n, col):
    from cudamica_b200.engine import AmicaError
    eng, rng = _engine(n, 2)
    with eng:
        A = np.stack([synth.mixing_matrix(rng, n, 50.0) for _ in range(2)])
        good = A.copy()
        A[1, col] = 0.0
        eng.set_params(A=A)
        with pytest.raises(AmicaError) as e:
            eng.estep_stats()
        assert e.value.code == -22
        eng.set_params(A=good)              # and the context goes on
        assert np.isfinite(eng.estep_stats()).all()
