"""The E-step's sums over the kept samples only, in every fused form and lane packing
(1, 2 and 4 sample sets; one and several models; with the split correction of phi),
against the FP64 oracle given the same mask.  Tolerances as where no sample is
dropped (test_tile_shapes_gpu.py, test_plain_shapes_gpu.py): the LL to 2e-6 nats per
sample and channel, the sums to 2e-4 (mixed) and 2e-5 (FP32) of their largest entries."""
import numpy as np
import pytest

from oracle import oracle as O
from test_parity_headline_gpu import _as_stored, _errs
from test_tile_shapes_gpu import _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,T,M,m,precision,kw", [
    (20, 30_001, 1, 3, 1, {}), (40, 30_002, 1, 4, 1, {}), (100, 20_003, 1, 2, 1, {}), (64, 20_001, 1, 5, 1, {}),
    (20, 30_003, 2, 2, 1, {}), (40, 30_001, 3, 3, 1, {}), (128, 20_002, 2, 3, 1, {}), (100, 20_001, 2, 5, 1, {}),
    (32, 30_001, 1, 3, 1, {"phi_split": 1}), (64, 20_003, 2, 3, 1, {"phi_split": 1}),
    (71, 20_001, 2, 3, 0, {}), (32, 20_003, 1, 1, 0, {})])
def test_sums_over_the_kept_samples(n, T, M, m, precision, kw):
    from cudamica_b200.engine import Amica
    xs, means, S, ldetS, A0, c0 = _data(n, T, M, m)
    orc = O.Oracle(_as_stored(xs, precision), M, m, A0, c0, ldetS, nthreads=8)
    orc.prepare()
    with Amica(n, T, M, m, precision=precision, rejsig=0.5, **kw) as e:
        e.set_sphered(xs, means, S, ldetS)
        e.init(A0, c0)
        full = e.estep_stats()
        for _ in range(2):
            dropped = e.reject_now()
            assert dropped > T // 20
            e.estep_stats()
        keep = e.loglik()[2]
        got = e.estep_stats()
    orc.keep[:] = keep
    want = orc.estep()
    kept = int(keep.sum())
    assert kept < 0.8 * T and got[0] != full[0]
    assert abs(got[0] - want[0]) / (n * T) < 2e-6
    errs = _errs(got, want, n, M, m)
    for k in ("vs", "cn", "s2", "us", "kn", "ln", "bd", "rn", "phi"):
        assert errs[k] < (2e-4 if precision else 2e-5), (k, errs[k])


@pytest.mark.parametrize("m", [1, 3, 4, 5])
def test_cohort_leaves_the_parameters_of_each_fit_alone(m):
    """Every sum goes through the parameters after an iteration.  The samples' terms
    are the same as in a fit alone, their FP32 sums grouped differently: a few 1e-7 of
    the sums, and of the parameters made from them."""
    from cudamica_b200 import synth
    from cudamica_b200.engine import Amica, PersistentCohort
    cohort, alone = [], []
    for n, T in ((12, 3001), (40, 9000), (90, 7001), (128, 40)):
        x = np.random.default_rng(n).laplace(size=(T, n)).astype(np.float32)
        if T < n:
            x = np.random.default_rng(n).laplace(size=(T, n)).astype(np.float64)
        for fits in (cohort, alone):
            e = Amica(n, T, 1, m)
            if T < n:
                e.set_sphered(x)
            else:
                e.load_data(x)
                e.preprocess()
            e.init(*synth.norand_init(n, 1))
            fits.append(e)
    PersistentCohort(cohort).run(1)
    for a, b in zip(cohort, alone):
        b.run(1)
        pa, pb = a.params(), b.params()
        for k in ("A", "c", "gm", "alpha", "mu", "beta", "rho"):
            assert np.linalg.norm(pa[k] - pb[k]) <= 1e-5 * max(np.linalg.norm(pb[k]), 1e-2 * np.sqrt(a.n)), k


@pytest.mark.parametrize("n,T,M,m", [(5, 47, 1, 1), (33, 97, 1, 4), (65, 49, 1, 3), (128, 48, 1, 5), (5, 47, 2, 3),
                                     (65, 49, 2, 2), (128, 1, 2, 1)])
def test_sums_of_one_and_two_tiles(n, T, M, m):
    """A few samples: phi's TF32 operands, each within 2^-11, do not average out, so its
    error is up to 2^-10 of sum |g b|, about twice its largest entry; the others as above."""
    from cudamica_b200 import synth
    from cudamica_b200.engine import Amica
    T = max(T, 2)
    xs = 2.0 * np.random.default_rng(n).laplace(size=(T, n)) / np.sqrt(2.0)
    A0, c0 = synth.norand_init(n, M)
    orc = O.Oracle(_as_stored(xs, 1), M, m, A0, c0, 0.0, nthreads=4)
    orc.prepare()
    want = orc.estep()
    with Amica(n, T, M, m, precision=1) as e:
        e.set_sphered(xs)
        e.init(A0, c0)
        got = e.estep_stats()
    a, b = O.split_stats(got, n, M, m), O.split_stats(want, n, M, m)
    for k, tol in (("vs", 2e-4), ("us", 2e-4), ("s2", 2e-4), ("phi", 2e-3)):
        for h in range(M):
            assert np.abs(a[k][h] - b[k][h]).max() < tol * np.abs(b[k][h]).max(), k
