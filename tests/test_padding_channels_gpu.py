"""Padding channels (a form works on 32, 64 or 128 per sample) add exactly 0 to a
sample's log-likelihood in every fused form: the one-model kernel, the one with the
split correction of phi, and the several-model kernel with two models of the same
parameters give the same Lt.

The forms round a channel's log-sum-exp differently, by at most 2^-22 (log2 units)
and independently, so a sample's difference is of the order of sqrt(n) 2^-22 and the
mean over thousands of samples far below that, which is the bound here.  A padding
channel that adds one unit in the last place (2^-23) is one-sided and stays in the mean:
30 to 63 of them are above the bound."""
import numpy as np
import pytest

from cudamica_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,T", [(2, 8001), (3, 8002), (33, 8001), (65, 8003)])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5])
def test_padding_channels_add_nothing(n, T, m):
    from cudamica_b200.engine import Amica
    xs = np.random.default_rng(n).laplace(size=(T, n))
    A0, c0 = synth.norand_init(n, 1)
    Lt = {}
    for name, M, kw in (("one", 1, {}), ("split", 1, {"phi_split": 1}), ("two", 2, {}),
                        ("two, split", 2, {"phi_split": 1})):
        with Amica(n, T, M, m, precision=1, **kw) as e:
            assert e.kernel == "tc_tf32"
            e.set_sphered(xs)
            e.init(np.concatenate([A0] * M), np.concatenate([c0] * M))
            p = e.params()
            p["gm"][:] = 1.0                       # the constant of Lt without log gm
            e.set_params(gm=p["gm"], **{k: np.repeat(p[k][:1], M, axis=0) for k in ("alpha", "mu", "beta", "rho")})
            e.estep_stats()
            Lt[name] = e.loglik()[0]
    for name in ("split", "two", "two, split"):
        for h in range(Lt[name].shape[0]):
            assert abs((Lt[name][h] - Lt["one"][0]).mean()) < np.sqrt(n) * 2.0 ** -22 * np.log(2.0), name
