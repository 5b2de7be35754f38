"""After a preprocessing that ended with an error (a bounded device wait that the test
hook lets run out) there are no sphered data: every call that needs them is out of
order until a preprocessing, or sphered data from the caller, has succeeded."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu


def test_nothing_iterates_on_the_scratch_of_a_failed_preprocessing():
    from cudamica_b200.engine import Amica, AmicaError
    n, T = 130, 3000
    x = np.random.default_rng(1).laplace(size=(T, n)).astype(np.float32)
    with Amica(n, T, 1, 2) as e:
        e.load_data(x)
        e.preprocess()
        e.init(*synth.norand_init(n, 1))
        want = e.step().ll
        e.init(*synth.norand_init(n, 1))
        e.arm_wait_fault(1_000_000)
        with pytest.raises(AmicaError) as err:
            e.preprocess()
        assert err.value.code == -24
        for call in (e.step, lambda: e.run(1), e.estep_stats, e.adjoint, e.sphere, e.time_estep):
            with pytest.raises(AmicaError) as err:
                call()
            assert err.value.code == -21
        e.preprocess()
        assert e.step().ll == want
        e.arm_wait_fault(1_000_000)
        with pytest.raises(AmicaError):
            e.preprocess()
        e.set_sphered(x.astype(np.float64))
        assert np.isfinite(e.step().ll)
