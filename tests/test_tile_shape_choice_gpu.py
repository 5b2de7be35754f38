"""amica_set_tile_shape(ctx, 0) is the shape of 3 density warpgroups for every mixture
count (a new context starts in the default for its counts, which is another one with
five mixtures), told by its grid: 48-sample tiles.  A cohort runs its own shape,
whichever of the two its contexts are in."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,m", [(1, 3), (1, 4), (1, 5), (2, 5)])
@pytest.mark.parametrize("n,pack", [(20, 4), (40, 2), (100, 1)])
def test_every_shape_can_be_asked_for(n, pack, M, m):
    from cudamica_b200.engine import Amica
    T = 96 * pack                                # 2 tiles of 48 samples, 3 of 32
    with Amica(n, T, M, m, precision=1) as e:
        for shape, tiles in ((0, 2), (1, 3), (2, 3), (0, 2)):
            e.set_tile_shape(shape)
            assert e.set_grid(0) == tiles


@pytest.mark.parametrize("m", [3, 5])
def test_cohort_of_contexts_in_either_shape(m):
    from cudamica_b200.engine import Amica, PersistentCohort
    fits = []
    for shapes in ((None, None), (0, None), (0, 0)):
        engines = []
        for s, (n, T) in zip(shapes, ((12, 3001), (90, 7001))):
            e = Amica(n, T, 1, m, precision=1)
            e.load_data(np.random.default_rng(n).laplace(size=(T, n)).astype(np.float32))
            e.preprocess()
            e.init(*synth.norand_init(n, 1))
            if s is not None:
                e.set_tile_shape(s)
            engines.append(e)
        PersistentCohort(engines).run(2)
        fits.append([e.params() for e in engines])
        for e in engines:
            e.close()
    for other in fits[1:]:
        for a, b in zip(fits[0], other):
            for k in a:
                assert np.array_equal(a[k], b[k]), k          # the same kernel on the same tiles
