"""Calls between amica_run_async and amica_run_wait: the stream orders them behind
the batch, and what they return and leave is what the same calls give one after
another.  Bit for bit the same (one GPU, one order of every sum), so no tolerance."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu


def _fit():
    from cudamica_b200.engine import Amica
    n, T = 6, 5000
    e = Amica(n, T, 1, 2)
    e.load_data(np.random.default_rng(0).laplace(size=(T, n)).astype(np.float32))
    e.preprocess()
    e.init(*synth.norand_init(n, 1))
    return e


def _rec(r):
    return (r.iter, r.ll, r.lrate, r.newton, r.ll_decreased)


@pytest.mark.parametrize("batch", [1, 3, 300])                # 300: past the pinned records
def test_step_between_run_async_and_run_wait(batch):
    with _fit() as a, _fit() as b:
        want = [_rec(a.step()) for _ in range(batch + 2)]
        b.run_async(batch)
        between = _rec(b.step())
        assert [_rec(r) for r in b.run_wait()] == want[:batch]
        assert between == want[batch]
        assert _rec(b.run(1)[0]) == want[batch + 1]
        assert np.array_equal(a.params()["A"], b.params()["A"])


def test_set_iter_state_between_run_async_and_run_wait():
    with _fit() as a, _fit() as b:
        a.run(3)
        a.set_iter_state(20, 0.05, -9.0)
        want = [_rec(r) for r in a.run(2)]
        b.run_async(3)
        b.set_iter_state(20, 0.05, -9.0)
        b.run_wait()
        assert [_rec(r) for r in b.run(2)] == want and [w[0] for w in want] == [21, 22]


def test_init_between_run_async_and_run_wait():
    with _fit() as a, _fit() as b:
        want = [_rec(a.step()) for _ in range(2)]
        b.run_async(5)
        b.init(*synth.norand_init(6, 1))
        b.run_wait()
        assert [_rec(r) for r in b.run(2)] == want


def test_rolled_back_batch_leaves_its_first_iteration_number():
    from cudamica_b200.engine import AmicaError
    with _fit() as e:
        e.run(4)
        good = e.params()
        e.set_params(mu=np.full_like(good["mu"], np.nan))
        with pytest.raises(AmicaError) as err:
            e.run(3)
        assert err.value.code == -23
        e.set_params(mu=good["mu"])
        assert e.step().iter == 5
