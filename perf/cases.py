"""Performance cases of the AMICA engine: what a user's program has it do.

Every case goes through the package's public entry points
(``cudamica_b200.engine``).  The kinds are

* ``iterate``: one EM iteration of a resumed fit: parameters and loop state in
  (``set_params``, ``set_iter_state``), ``run(1)`` on the data that is resident
  on the GPU, parameters out.  The inner loop of every fit; both precisions.
* ``reject``: the first iteration of a fit with sample rejection on, with the
  per-sample likelihoods and the keep mask read back (``loglik``).
* ``fit``: a whole short call: raw data from device memory, sphering, initial
  state, one iteration, parameters out.
* ``preprocess``: raw data from device memory, centring and sphering.
* ``adjoint``: the log-likelihood and its gradient.
* ``noalloc``: the allocation-free E-step of an on-line caller.
* ``cohort``: one iteration of several single-model fits advanced together.

The data follow the package's synthetic recipes: generalized-Gaussian sources
(shape 1 to 2.5) mixed by ill-conditioned matrices, the generating model
switching in contiguous blocks of 500 to 2500 samples when there are several.
``iterate`` starts from a state of the middle of a fit: mixing matrices near the
generating ones, so that the models' responsibilities are as concentrated as
they are after the first iterations.

One iteration and not many makes up a pass because the EM map multiplies a
last-bit difference by 10 to 100 per iteration.  Parameters, statistics and
gradients are ratios and sums of terms evaluated in FP32 (or from TF32
products) that the interface hands out as FP64; they are returned here in FP32,
the precision that they carry.  A model's mixing columns and its centre c come
as one affine map (x = A s + c): c is a mean of centred data, and for a single
model 0 but for rounding.  The sphering is FP64 throughout and is returned as
it comes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cudamica_b200.engine import Amica, PersistentCohort, estep_stats_noalloc

PARAMS = ("W", "gm", "alpha", "mu", "beta", "rho")
LRATE0, ITER0 = 0.1, 100          # an iteration past the start of the Newton steps
COHORT_N = (32, 64, 128)


def listed():
    return [
        # an on-line caller's E-step over a few seconds of data: the smallest call
        dict(name="noalloc_n32_t4k", kind="noalloc", n=32, T=4096, M=1, m=3),
        # the small single-model recording of the golden tests
        dict(name="iter_n32_t60k", kind="iterate", n=32, T=60_000, M=1, m=3, precision=1),
        # odd channel and sample counts, several models, two mixtures
        dict(name="iter_n19_t30011_M2", kind="iterate", n=19, T=30_011, M=2, m=2, precision=1),
        # the EEG-scale single-model fit
        dict(name="iter_n64_t500k", kind="iterate", n=64, T=500_000, M=1, m=3, precision=1),
        # the benchmark's workload: three models at 128 channels
        dict(name="iter_n128_t1m_M3", kind="iterate", n=128, T=1_000_000, M=3, m=3, precision=1),
        # the FP32 form, ragged
        dict(name="iter_fp32_n71_t200003_M2", kind="iterate", n=71, T=200_003, M=2, m=3, precision=0),
        # high-density recordings above 128 channels, four models of five mixtures
        dict(name="iter_n256_t400k_M4", kind="iterate", n=256, T=400_000, M=4, m=5, precision=1),
        # outlier rejection in an EEG-scale fit
        dict(name="reject_n64_t300k", kind="reject", n=64, T=300_000, M=1, m=3, precision=1),
        # sphering at the benchmark's size, and a whole short call above 128 channels
        dict(name="preprocess_n128_t1m", kind="preprocess", n=128, T=1_000_000, M=1, m=3, precision=1),
        dict(name="fit_n160_t50k", kind="fit", n=160, T=50_000, M=1, m=3, precision=1),
        # the gradient for a user's own optimiser
        dict(name="adjoint_n100_t120k_M2", kind="adjoint", n=100, T=120_000, M=2, m=3, precision=1),
        # several recordings at once
        dict(name="cohort_6", kind="cohort", subjects=6, T=100_000, T_hi=800_000, m=3),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate"] * 8 + ["reject", "preprocess", "fit", "adjoint", "noalloc", "cohort"])
    if kind == "cohort":
        lo = _log_uniform(rng, 20_000, 200_000)
        return dict(kind=kind, subjects=rng.randint(2, 6), T=lo, T_hi=4 * lo, m=rng.randint(1, 5))
    m = rng.randint(1, 5)
    if kind == "noalloc":
        return dict(kind=kind, n=_log_uniform(rng, 8, 128), T=_log_uniform(rng, 1000, 16_000), M=rng.randint(1, 2), m=m)
    n = _log_uniform(rng, 16, 256)
    M = rng.choice([1, 1, 2, 3, 4])
    precision = 0 if kind == "iterate" and rng.random() < 0.2 else 1
    # the work of a pass grows with n M m T; the FP32 form costs about four times as much per sample
    most = 1.1e9 / (n * M * m) / (4 if precision == 0 or n > 128 else 1)
    return dict(kind=kind, n=n, T=_log_uniform(rng, 20_000, max(40_000, min(1_000_000, most))), M=M, m=m,
                precision=precision)


# ------------------------------------------------------------------ inputs
def _data(n, T, M, seed):
    """Raw data (T x n FP32 on the GPU) and the generating mixing matrices."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = np.random.default_rng(seed)
    rho = torch.rand(n, generator=g, device="cuda") * 1.5 + 1.0
    s = torch._standard_gamma((1.0 / rho).expand(T, n).contiguous(), generator=g).clamp_(min=1e-30)
    s.pow_(1.0 / rho)
    s.mul_(torch.randint(0, 2, (T, n), generator=g, device="cuda", dtype=torch.int8) * 2 - 1)
    s.div_(torch.exp(0.5 * (torch.lgamma(3.0 / rho) - torch.lgamma(1.0 / rho))))
    mixing = []
    for _ in range(M):
        q = [torch.linalg.qr(torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64))[0] for _ in range(2)]
        sv = torch.logspace(0.0, -math.log10(30.0), n, device="cuda", dtype=torch.float64)
        mixing.append((q[0] * sv) @ q[1].T)
    if M == 1:
        x = s @ mixing[0].float().T
    else:
        lengths = r.integers(500, 2501, T // 500 + 1)
        models = np.cumsum(np.concatenate([[0], 1 + r.integers(0, M - 1, lengths.size - 1)])) % M
        label = torch.from_numpy(np.repeat(models, lengths)[:T]).cuda()
        x = torch.empty_like(s)
        for h in range(M):
            at = (label == h).nonzero(as_tuple=True)[0]
            x[at] = s[at] @ mixing[h].float().T
    x += 0.03 * torch.randn(T, n, generator=g, device="cuda")
    return x, mixing


def _chunks(T, width):
    step = max(1, int(5e7 // width))
    return [(t, min(T, t + step)) for t in range(0, T, step)]


def _sphering(x):
    """mean, S = 2 C^(-1/2) and -log|det S| in 64 bits."""
    T, n = x.shape
    mean = sum(x[a:b].double().sum(0) for a, b in _chunks(T, n)) / T
    C = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    for a, b in _chunks(T, n):
        xc = x[a:b].double() - mean
        C += xc.T @ xc
    d, V = torch.linalg.eigh(C / T)
    S = (V * (2.0 / d.sqrt())) @ V.T
    return mean, S, -torch.log(2.0 / d.sqrt()).sum()


def _mid_fit(n, M, m, mixing, S, seed):
    """Parameters of the middle of a fit (host FP64, the engine's storage order)."""
    r = np.random.default_rng(seed + 77)
    S = S.cpu().numpy()
    p = {k: np.empty((M, m, n)) for k in ("alpha", "mu", "beta", "rho")}
    A, c = np.empty((M, n, n)), 0.02 * r.standard_normal((M, n))
    for h in range(M):
        a = S @ mixing[h].cpu().numpy()
        scale = np.linalg.norm(a, axis=0)
        a = a / scale + 0.02 / math.sqrt(n) * r.standard_normal((n, n))
        A[h] = (a / np.linalg.norm(a, axis=0)).T            # column-major
        w = np.exp(0.5 * r.standard_normal((m, n)))
        p["alpha"][h] = w / w.sum(0)
        p["mu"][h] = 0.3 * r.standard_normal((m, n)) * scale
        p["beta"][h] = np.exp(r.uniform(math.log(0.7), math.log(2.0), (m, n))) / scale ** 2
        p["rho"][h] = r.uniform(1.05, 1.95, (m, n))
    return dict(A=A, c=c, gm=np.full(M, 1.0 / M), **p)


def _start(n, M, seed):
    """A fit's first state: A near the identity with unit columns."""
    r = np.random.default_rng(seed + 5)
    a = np.eye(n) + 0.05 * (r.random((M, n, n)) - 0.5)
    return a / np.linalg.norm(a, axis=2, keepdims=True), 0.1 * r.standard_normal((M, n))


def _engine(case, x):
    rej = dict(do_reject=1, rejstart=1, rejint=1) if case["kind"] == "reject" else {}
    e = Amica(x.shape[1], x.shape[0], case.get("M", 1), case["m"], precision=case.get("precision", 1), **rej)
    torch.cuda.synchronize()                                 # x is ready for the engine's own stream
    e.load_data_device(x.data_ptr())
    return e


def _cohort_shapes(case):
    k = case["subjects"]
    return [(COHORT_N[i % 3], int(case["T"] + (case["T_hi"] - case["T"]) * (i * 5 % k) / max(1, k - 1)) + i)
            for i in range(k)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cohort":
        engines, params = [], []
        for i, (n, T) in enumerate(_cohort_shapes(case)):
            x, mixing = _data(n, T, 1, seed * 64 + i)
            e = _engine(case, x)
            e.preprocess()
            p = _mid_fit(n, 1, case["m"], mixing, _sphering(x)[1], seed * 64 + i)
            e.init(p["A"], p["c"])
            engines.append(e)
            params.append(p)
        return dict(kind=kind, engines=engines, params=params, cohort=PersistentCohort(engines))
    n, T, M, m = case["n"], case["T"], case["M"], case["m"]
    x, mixing = _data(n, T, M, seed)
    if kind == "noalloc":
        mean, S, ldet = _sphering(x)
        p = _mid_fit(n, M, m, mixing, S, seed)
        width = next(w for w in (32, 64, 128, 256) if n <= w)
        xs = torch.zeros(T, width, device="cuda")
        xs[:, :n] = ((x.double() - mean) @ S.T).float()
        d = {k: torch.from_numpy(v).cuda() for k, v in p.items()}
        size = 1 + 2 * n + n * n + 7 * m * n
        return dict(kind=kind, case=case, x=xs, p=d, ldet=float(ldet),
                    stats=torch.zeros(1 + M * size, dtype=torch.float64, device="cuda"))
    e = _engine(case, x)
    s = dict(kind=kind, case=case, engine=e)
    if kind in ("preprocess", "fit"):
        s["x"] = x
    else:
        e.preprocess()
    if kind in ("reject", "fit"):
        s["A0"], s["c0"] = _start(n, M, seed)
    if kind in ("iterate", "adjoint"):
        s["params"] = _mid_fit(n, M, m, mixing, _sphering(x)[1], seed)
        e.init(s["params"]["A"], s["params"]["c"])
        e.set_params(**s["params"])
    return s


# ------------------------------------------------------------------ the passes
def _out(e, records):
    p = {k: v.astype(np.float32) for k, v in e.params().items()}
    return dict({k: p[k] for k in PARAMS}, affine=np.concatenate([p["A"], p["c"][:, None]], 1),
                ll=np.float32([r.ll for r in records]))


def _resume(e, p):
    e.set_params(**p)
    e.set_iter_state(ITER0, LRATE0, -1e3)


def run(state):
    kind = state["kind"]
    if kind == "cohort":
        for e, p in zip(state["engines"], state["params"]):
            _resume(e, p)
        records, _ = state["cohort"].run(1)
        return [_out(e, r) for e, r in zip(state["engines"], records)]
    if kind == "noalloc":
        case, d = state["case"], state["p"]
        n, T, M, m = case["n"], case["T"], case["M"], case["m"]
        estep_stats_noalloc(state["x"].data_ptr(), state["x"].shape[1], n, T, M, m, d["A"].data_ptr(),
                            d["c"].data_ptr(), d["alpha"].data_ptr(), d["mu"].data_ptr(), d["beta"].data_ptr(),
                            d["rho"].data_ptr(), d["gm"].data_ptr(), state["ldet"], state["stats"].data_ptr(),
                            stream=torch.cuda.current_stream().cuda_stream)
        return _sections(state["stats"].float(), n, M, m)
    e = state["engine"]
    if kind == "iterate":
        _resume(e, state["params"])
        return _out(e, e.run(1))
    if kind == "reject":
        e.init(state["A0"], state["c0"])
        records = e.run(1)
        Lt, P, keep = e.loglik()
        return dict(_out(e, records), Lt=Lt.astype(np.float32), P=P.astype(np.float32), keep=keep,
                    rejected=int(records[0].nrejected))
    if kind == "preprocess":
        e.load_data_device(state["x"].data_ptr())
        e.preprocess()
        return e.sphere()
    if kind == "fit":
        e.load_data_device(state["x"].data_ptr())
        e.preprocess()
        e.init(state["A0"], state["c0"])
        return _out(e, e.run(1))
    ll, grads = e.adjoint()
    return dict({k: v.astype(np.float32) for k, v in grads.items()}, ll=np.float32([ll]))


def _sections(v, n, M, m):
    """The flat statistics vector by quantity (views)."""
    w, k = v[1:].reshape(M, -1), m * n
    at = 1 + 2 * n + n * n
    d = dict(ll=v[:1], moments=w[:, :1 + n], s2=w[:, 1 + n:1 + 2 * n], phi=w[:, 1 + 2 * n:at])
    for i, q in enumerate(("us", "kn", "ln", "mn", "md", "bd", "rn")):
        d[q] = w[:, at + i * k:at + (i + 1) * k]
    return d


# ------------------------------------------------------------------ what a pass cannot do without
def _em_work(n, T, M, m):
    """The data once, the per-sample likelihoods once, the two contractions and
    about 40 operations per sample, channel, model and mixture."""
    return 4.0 * T * (n + M + 1), T * M * (4.0 * n * n + 40.0 * m * n)


def work(case):
    kind = case["kind"]
    if kind == "cohort":
        w = [_em_work(n, T, 1, case["m"]) for n, T in _cohort_shapes(case)]
        return dict(bytes=sum(b for b, _ in w), flops=sum(f for _, f in w))
    n, T, M, m = case["n"], case["T"], case["M"], case["m"]
    # sphering: raw data twice (the covariance needs the mean only as a correction), sphered data out
    sphere = (12.0 * T * n, 3.0 * T * n * n)
    if kind == "preprocess":
        return dict(bytes=sphere[0], flops=sphere[1])
    b, f = _em_work(n, T, M, m)
    if kind == "fit":
        b, f = b + sphere[0], f + sphere[1]
    if kind == "reject":
        b += 5.0 * T                                         # P and the mask again
    if kind == "noalloc":
        b = 4.0 * T * n + 8.0 * (1 + M * (1 + 2 * n + n * n + 7 * m * n))
    return dict(bytes=b, flops=f)


# ------------------------------------------------------------------ the same in 64 bits
def _estep(x, p, ldet):
    """Sums of the E-step over the sphered data x (64 bits), and per-sample Lt, P."""
    T, n = x.shape
    M, m, _ = p["mu"].shape
    z = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")  # noqa: E731
    W = torch.linalg.inv(p["A"].transpose(1, 2))             # W[h] = W_h
    q = {k: z(M, m, n) for k in ("us", "kn", "ln", "mn", "md", "bd", "rn")}
    q |= dict(vsum=z(M), s2=z(M, n), phi=z(M, n, n), gx=z(M, n, n), vx=z(M, n), Lt=z(M, T), P=z(T), W=W)
    r, sb = p["rho"], p["beta"].sqrt()
    const = p["alpha"].log() + 0.5 * p["beta"].log() - math.log(2.0) - torch.lgamma(1.0 + 1.0 / r)
    base = p["gm"].log() + torch.linalg.slogdet(W)[1] + ldet
    for a, e in _chunks(T, n * m):
        for h in range(M):
            b = (x[a:e] - p["c"][h]) @ W[h].T
            y = sb[h] * (b[:, None, :] - p["mu"][h])
            q["Lt"][h, a:e] = base[h] + torch.logsumexp(const[h] - y.abs() ** r[h], 1).sum(1)
    q["P"][:] = torch.logsumexp(q["Lt"], 0)
    for a, e in _chunks(T, n * m):
        for h in range(M):
            xc = x[a:e] - p["c"][h]
            b = xc @ W[h].T
            y = sb[h] * (b[:, None, :] - p["mu"][h])
            ay = y.abs()
            pw = ay ** r[h]
            v = (q["Lt"][h, a:e] - q["P"][a:e]).exp()
            u = torch.softmax(const[h] - pw, 1) * v[:, None, None]
            f = torch.where(ay > 0, r[h] * pw / torch.where(ay > 0, y, torch.ones_like(y)), torch.zeros_like(y))
            big = r[h] > 2.0
            q["us"][h] += u.sum(0)
            q["kn"][h] += p["beta"][h] * (u * f * f).sum(0)
            q["ln"][h] += (u * (f * y - 1.0) ** 2).sum(0)
            q["mn"][h] += (u * f).sum(0)
            per = torch.where(ay > 0, f / torch.where(ay > 0, y, torch.ones_like(y)), torch.zeros_like(y))
            q["md"][h] += sb[h] * (u * torch.where(big, f * f, per)).sum(0)
            q["bd"][h] += torch.where(big, r[h] * (u * pw).sum(0), (u * f * y).sum(0))
            q["rn"][h] += (u * torch.where(pw > 0, pw * pw.clamp(min=1e-300).log(), pw)).sum(0)
            g = (sb[h] * u * f).sum(1)
            q["phi"][h] += g.T @ b
            q["gx"][h] += g.T @ xc
            q["vsum"][h] += v.sum()
            q["s2"][h] += (v[:, None] * b * b).sum(0)
            q["vx"][h] += (v[:, None] * x[a:e]).sum(0)
    return q


def _mstep(q, p, T, it, lrate):
    """One M-step with the engine's defaults; `it` is the iteration's number."""
    M, m, n = p["mu"].shape
    vs = q["vsum"][:, None]
    alpha = q["us"] / vs[:, None]
    sig2 = q["s2"] / vs
    dk = q["kn"] / q["us"]
    kappa = (alpha * dk).sum(1)
    lam = (alpha * (p["mu"] ** 2 * dk + q["ln"] / q["us"])).sum(1)
    mu = p["mu"] + q["mn"] / q["md"]
    beta = p["beta"] * torch.where(p["rho"] > 2.0, torch.zeros_like(p["rho"]), q["us"]) / q["bd"]
    rho = p["rho"]
    rho = (rho + 0.1 * (1.0 - rho / torch.digamma(1.0 + 1.0 / rho) * q["rn"] / q["us"])).clamp(1.0, 2.0)
    ks = kappa * sig2
    ok = [bool((torch.outer(k, k) > 1.0).all()) for k in ks]
    newton = [it >= 50 and o for o in ok]
    lrate = min(1.0 if all(newton) else 0.1, lrate + min(0.1, lrate))
    A, eye = p["A"].transpose(1, 2), torch.eye(n, dtype=torch.float64, device="cuda")
    out = torch.empty_like(A)
    shift = torch.empty_like(p["c"])
    cnew = q["vx"] / vs
    for h in range(M):
        pr = q["phi"][h] / q["vsum"][h]
        if newton[h]:
            off = torch.outer(ks[h], ks[h]) - 1.0
            B = (torch.outer(sig2[h], kappa[h]) * pr - pr.T) / off
            B = torch.where(eye > 0, torch.diag((1.0 - pr.diagonal()) / lam[h]), B)
            out[h] = A[h] + lrate * A[h] @ B
        else:
            out[h] = A[h] - lrate * A[h] @ (eye - pr)
        shift[h] = q["W"][h] @ (cnew[h] - p["c"][h])
    norm = out.norm(dim=1)
    A = (out / norm[:, None, :]).transpose(1, 2)
    return dict(affine=torch.cat([A, cnew[:, None]], 1), W=q["W"].transpose(1, 2).contiguous(), gm=q["vsum"] / T, alpha=alpha,
                mu=mu * norm[:, None, :] - shift[:, None, :], beta=beta / norm[:, None, :] ** 2, rho=rho,
                ll=(q["P"].sum() / (n * T)).reshape(1))


def _first_params(A0, c0, m):
    """The engine's deterministic start: alpha = 1/m, mu spread, beta 1, rho 1.5."""
    M, n = c0.shape
    one = np.ones((M, m, n))
    mu = one * (np.arange(m) - (m - 1) / 2.0)[None, :, None]
    return dict(A=A0, c=c0, gm=np.full(M, 1.0 / M), alpha=one / m, mu=mu, beta=one, rho=1.5 * one)


def _cuda(p):
    return {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in p.items()}


def _exact_iterate(x, mixing, m, seed, M, case_kind):
    n = x.shape[1]
    mean, S, ldet = _sphering(x)
    if case_kind in ("reject", "fit"):
        p, it = _cuda(_first_params(*_start(n, M, seed), m)), 1
    else:
        p, it = _cuda(_mid_fit(n, M, m, mixing, S, seed)), ITER0 + 1
    xs = (x.double() - mean) @ S.T
    q = _estep(xs, p, ldet)
    return q, p, _mstep(q, p, x.shape[0], it, LRATE0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "cohort":
        out = []
        for i, (n, T) in enumerate(_cohort_shapes(case)):
            x, mixing = _data(n, T, 1, seed * 64 + i)
            o = _exact_iterate(x, mixing, case["m"], seed * 64 + i, 1, kind)[2]
            out.append(dict(o, mu=None))
        return out
    n, T, M, m = case["n"], case["T"], case["M"], case["m"]
    x, mixing = _data(n, T, M, seed)
    if kind == "preprocess":
        mean, S, ldet = _sphering(x)
        return S, mean, float(ldet)
    if kind == "noalloc":
        mean, S, ldet = _sphering(x)
        p = _cuda(_mid_fit(n, M, m, mixing, S, seed))
        q = _estep(((x.double() - mean) @ S.T).float().double(), p, ldet)
        d = {k: q[k].reshape(M, -1) for k in ("s2", "us", "kn", "ln", "mn", "bd", "rn")}
        # md, the mu denominator, is dominated by the samples nearest a kink of the density: no
        # FP32 value of it is near the 64-bit one (nor of mu, which is divided by it)
        return dict(d, ll=q["P"].sum().reshape(1), moments=torch.cat([q["vsum"][:, None], q["vx"]], 1),
                    phi=q["phi"].transpose(1, 2).reshape(M, -1), md=None)
    q, p, o = _exact_iterate(x, mixing, m, seed, M, "iterate" if kind == "adjoint" else kind)
    if kind == "adjoint":
        r, k = p["rho"], 1.0 / (n * T)
        A = p["A"].transpose(1, 2)
        dW = q["vsum"][:, None, None] * A.transpose(1, 2) - q["gx"]           # dL/dW_h(i, k)
        dbeta = (q["us"] - q["bd"]) / (2.0 * p["beta"])
        drho = q["us"] * torch.digamma(1.0 + 1.0 / r) / r ** 2 - q["rn"] / r
        return dict(W=dW.transpose(1, 2).contiguous() * k, mu=p["beta"].sqrt() * q["mn"] * k, beta=dbeta * k,
                    rho=drho * k, ll=o["ll"])
    o = dict(o, mu=None)
    if kind == "reject":
        # the mask is a comparison of FP32 values with their own threshold: no 64-bit value
        o |= dict(Lt=q["Lt"], P=q["P"], keep=None, rejected=None)
    return o
