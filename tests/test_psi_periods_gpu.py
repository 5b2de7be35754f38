"""Psi = sum g x^T of the split form (above 128 channels), accumulated in tensor memory
over periods of 64 to 128 blocks of 32 samples and added up in FP64: a long fit
against the sum of sixteen contexts with a sixteenth of its samples each, whose
periods are short.  The products are the same, only their sum is grouped
differently; with A near the identity phi's large entries are sums of one sign.

An MMA step (four a block) loses about one last place of its running sum, always
towards 0: at most 2^-23 of a sum that is on average half of what it ends at, 2^-24
a step of a period."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu


def _phi(xs, n, M, m, A0, c0):
    from cudamica_b200.engine import Amica
    with Amica(n, xs.shape[0], M, m, precision=1) as e:
        assert e.kernel == "split_tf32"
        e.set_sphered(xs)
        e.init(A0, c0)
        v = e.estep_stats()
    return v[1:].reshape(M, -1)[:, 1 + 2 * n:1 + 2 * n + n * n]


# blocks a chunk (148 SMs, 2 M halves): past two full periods, one block past one
# period, no second period
@pytest.mark.parametrize("n,M,m,blocks", [(130, 2, 1, 256), (160, 4, 2, 129), (256, 4, 1, 64)])
def test_psi_of_long_chunks(n, M, m, blocks):
    T = 148 // (2 * M) * 32 * blocks - 7
    xs = np.random.default_rng(n).laplace(size=(T, n))
    A0, c0 = synth.norand_init(n, M)
    whole = _phi(xs, n, M, m, A0, c0)
    parts = sum(_phi(p, n, M, m, A0, c0) for p in np.array_split(xs, 16))
    period = min(max((blocks + 1) // 2, 64), 128)
    for h in range(M):
        assert np.linalg.norm(whole[h] - parts[h]) < 4 * period * 2.0 ** -24 * np.linalg.norm(parts[h])
