"""The single-model E-step kernel at the edges of its tiles and lane packings
(1, 2 and 4 sample sets; partial tiles, one tile, more tiles than CTAs, dropped
samples), every mixture count, alone and in a cohort, against the FP64 oracle on
the data as the mixed form stores it.  Tolerances as for the other shapes of the
mixed form (test_tile_shapes_gpu.py): the LL to 2e-6 nats per sample and
channel, the sums to 2e-4 of their largest entries."""
import numpy as np
import pytest

from oracle import oracle as O
from test_parity_headline_gpu import _as_stored, _errs
from test_tile_shapes_gpu import _data

pytestmark = pytest.mark.gpu


def _check(s, s_orc, n, T, m):
    assert abs(s[0] - s_orc[0]) / (n * T) < 2e-6
    errs = _errs(s, s_orc, n, 1, m)
    for k in ("vs", "cn", "s2", "us", "kn", "ln", "bd", "rn", "phi"):
        assert errs[k] < 2e-4, (k, errs[k])


@pytest.mark.parametrize("n,T,m", [(5, 47, 1), (31, 193, 2), (32, 60_001, 3), (33, 97, 4), (64, 48 * 148 * 2 + 1, 5),
                                   (65, 49, 3), (128, 48 * 148 + 47, 4), (100, 30_011, 1)])
def test_single_model_estep_matches_the_oracle(n, T, m):
    from cudamica_b200.engine import Amica
    xs, means, S, ldetS, A0, c0 = _data(n, T, 1, m) if T > 1000 else _small(n, T)
    orc = O.Oracle(_as_stored(xs, 1), 1, m, A0, c0, ldetS, nthreads=8)
    orc.prepare()
    want = orc.estep()
    with Amica(n, T, 1, m, precision=1) as eng:
        eng.set_sphered(xs, means, S, ldetS)
        eng.init(A0, c0)
        for shape in (0, 1, 2):
            eng.set_tile_shape(shape)
            s = eng.estep_stats()
            if T > 1000:
                _check(s, want, n, T, m)
            else:                        # few samples: c and single sums are rounding noise
                assert abs(s[0] - want[0]) / (n * T) < 2e-6
                assert s[1] == want[1] == T
            P = eng.loglik()[1]
            assert abs(P.sum() - s[0]) < 1e-6 * abs(s[0])


def _small(n, T):
    from cudamica_b200 import synth
    rng = np.random.default_rng(n)
    xs = 2.0 * rng.laplace(size=(T, n)) / np.sqrt(2.0)
    A0, c0 = synth.norand_init(n, 1)
    return xs, np.zeros(n), 2.0 * np.eye(n), -n * np.log(2.0), A0, c0


@pytest.mark.parametrize("m", [2, 5])
def test_cohort_of_one_model_fits_matches_each_alone(m):
    from cudamica_b200 import synth
    from cudamica_b200.engine import Amica, PersistentCohort
    engines, alone = [], []
    for n, T in ((12, 3001), (40, 9000), (90, 7001)):
        x = np.random.default_rng(n).laplace(size=(T, n)).astype(np.float32)
        pair = []
        for _ in range(2):
            e = Amica(n, T, 1, m)
            e.load_data(x)
            e.preprocess()
            e.init(*synth.norand_init(n, 1))
            pair.append(e)
        engines.append(pair[0])
        alone.append(pair[1])
    records, _ = PersistentCohort(engines).run(1)
    for r, e in zip(records, alone):
        assert abs(r[0].ll - e.run(1)[0].ll) < 1e-6   # the same sums, grouped differently
