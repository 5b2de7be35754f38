"""The rejection pass at the edges of its 4096-sample chunks and past 256
chunks (one batch of the ordered sum over chunks), against the oracle's rule on
the same P: bit-exact, so no tolerance."""
import numpy as np
import pytest

from cudamica_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [200, 4095, 4096, 4097, 12289, 4096 * 257 + 5])
def test_reject_at_chunk_edges(T):
    from cudamica_b200.engine import Amica
    n = 4
    x = np.random.default_rng(T).laplace(size=(T, n)).astype(np.float32)
    with Amica(n, T, 1, 2, rejsig=2.5) as eng:
        eng.load_data(x)
        eng.preprocess()
        eng.init(*synth.norand_init(n, 1))
        keep = np.ones(T, dtype=np.uint8)
        for _ in range(2):                     # the second pass meets dropped samples
            eng.estep_stats()
            P = eng.p_relative().astype(np.float64)
            want, dropped, _, _ = O.reject(P, keep, 2.5)
            assert eng.reject_now() == dropped > 0
            keep = eng.loglik()[2].copy()
            assert np.array_equal(keep, want)
