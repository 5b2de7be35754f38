"""phi = sum g b^T of the several-model E-step: accumulated in tensor memory over
periods of 32 to 128 tiles and added up in FP64, at the edges of the periods (none,
one tile past one, whole ones, a short last one), in every lane packing and with the
split correction.

One cluster that runs every tile is compared with the full grid, whose CTAs run a
few tiles each: the products are the same, only their sum is grouped differently.
An MMA step rounds its running sum towards 0, by about one and at most some two
last places (2^-23) of a sum that is on average half of what it ends at: 2^-23 a
step of a period.  A tile of 48 rows has 6 steps (18 with the split correction)."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu


def _period(ntile):
    half = -(-((ntile + 1) // 2) // 16) * 16
    return min(max(half, 32), 128)


@pytest.mark.parametrize("n,M,m,ntile,kw", [
    (32, 2, 2, 32, {}), (32, 2, 2, 33, {}), (17, 3, 1, 64, {}), (64, 2, 3, 65, {}), (50, 2, 2, 97, {}),
    (128, 2, 1, 256, {}), (128, 3, 3, 257, {}), (128, 2, 3, 600, {}), (32, 2, 2, 1000, {}),
    (64, 2, 2, 513, {"phi_split": 1})])
def test_phi_of_one_cluster_matches_the_full_grid(n, M, m, ntile, kw):
    from cudamica_b200.engine import Amica
    pack = 4 if n <= 32 else 2 if n <= 64 else 1
    T = 48 * pack * ntile - 5
    x = np.random.default_rng(n).laplace(size=(T, n)).astype(np.float32)
    with Amica(n, T, M, m, precision=1, **kw) as e:
        e.load_data(x)
        e.preprocess()
        e.init(*synth.norand_init(n, M))
        full = e.estep_stats()
        assert e.set_grid(1) == 1
        one = e.estep_stats()
    size = 1 + 2 * n + n * n + 7 * m * n
    a, b = (v[1:].reshape(M, size)[:, 1 + 2 * n:1 + 2 * n + n * n] for v in (one, full))
    steps = 6 * min(ntile, _period(ntile)) * (3 if kw else 1)
    for h in range(M):
        assert np.linalg.norm(a[h] - b[h]) < steps * 2.0 ** -23 * np.linalg.norm(b[h])
    rest = np.ones(1 + M * size, bool)
    for h in range(M):
        rest[1 + h * size + 1 + 2 * n:1 + h * size + 1 + 2 * n + n * n] = False
    # the other sums go to FP64 every 16 tiles in either grid
    assert abs(one[0] - full[0]) < 1e-9 * abs(full[0])
    assert np.linalg.norm(one[rest] - full[rest]) < 1e-6 * np.linalg.norm(full[rest])
