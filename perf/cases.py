"""The work this library does for its users, as timed cases.

Families (a case's "path"):
  resample  the stand-alone primitives a filter of one's own calls at every
            observation: Resampler.reduce (ESS and log-weight sum), then the
            ancestors of the same log-weights
  filter    a whole filter run, BootstrapPF.filter (init, T steps, read-back),
            optionally with the path record and a sampled path
  step      the step-by-step API: init, then BootstrapPF.step per observation
  batch     many filters at once, BatchedBootstrapPF.filter: PMMH chains, SMC^2
            parameter particles, repeated likelihood estimates; optionally
            guided by a learned proposal
  train     training steps of the learned proposal, LearnedProposal.train

Sizes follow the repository's workloads (C1 plankton N = 4096 T = 100, C2
Lorenz-96 N = 65536 T = 200, C3 256 filters of 512..32768, C4 the guided
filter, C5 128 chains of 1024..8192) and the resampler harness (log-weights of
a shifted Gaussian, 16 particles upwards).
"""
import math

import numpy as np
import torch

from libbi_b200 import (BatchedBootstrapPF, BootstrapPF, MetropolisResampler, ModelL96, ModelPZ,
                        MultinomialResampler, SystematicResampler)
from libbi_b200.proposal import LearnedProposal

DEV = "cuda"
RESAMPLERS = {"systematic": SystematicResampler, "multinomial": MultinomialResampler,
              "metropolis": MetropolisResampler}
L96_DT, L96_H, L96_F, SIGMA_ETA, SIGMA_Y = 0.05, 0.01, 8.0, 0.1, 1.0
HIDDEN = 128


def listed():
    return [
        # a small filter's resampling on its own: launches and latency only
        dict(name="resample_small", path="resample", kind="systematic", n=1000, z=1.0, B=0, permute=True, offspring=True),
        # a filter too large for the caches, an odd size
        dict(name="resample_systematic_4m", path="resample", kind="systematic", n=4194301, z=2.0, B=0, permute=True,
             offspring=False),
        # the multinomial resampler, the reference's sorted form (not permuted)
        dict(name="resample_multinomial_1m", path="resample", kind="multinomial", n=1000003, z=2.0, B=0, permute=False,
             offspring=False),
        # Metropolis, 32 steps a particle
        dict(name="resample_metropolis_256k", path="resample", kind="metropolis", n=262144, z=1.0, B=32, permute=True,
             offspring=False),
        # C1: one plankton filter, resampled at every step
        dict(name="filter_pz_4096", path="filter", model="pz", dim=2, prec="f64", n=4096, T=100, kind="systematic", B=0,
             ess=1.0, paths=False),
        # C2: one Lorenz-96 filter
        dict(name="filter_l96_65536", path="filter", model="l96", dim=40, prec="f32", n=65536, T=200, kind="systematic",
             B=0, ess=0.5, paths=False),
        # the step API in the reference's default precision, a ragged size
        dict(name="step_l96_f64_20011", path="step", model="l96", dim=40, prec="f64", n=20011, T=1, kind="systematic",
             B=0, ess=0.5, paths=False),
        # C3: 256 Lorenz-96 filters of uneven sizes, mixed resamplers
        dict(name="batch_l96_256", path="batch", model="l96", prec="f32", nf=256, lo=512, hi=32768, T=100, ess=0.5,
             kind="mixed", guided=False),
        # C5: the filters of one PMMH iteration over 128 chains
        dict(name="batch_pz_128", path="batch", model="pz", prec="f64", nf=128, lo=1024, hi=8192, T=100, ess=1.0,
             kind="systematic", guided=False),
        # C4: 64 guided filters, the likelihood's deviation over seeds
        dict(name="guided_l96_64", path="batch", model="l96", prec="f32", nf=64, lo=4096, hi=4096, T=10, ess=0.5,
             kind="systematic", guided=True),
        # C5 with the learned proposal over the log-noise
        dict(name="guided_pz_128", path="batch", model="pz", prec="f64", nf=128, lo=1024, hi=8192, T=25, ess=1.0,
             kind="systematic", guided=True),
        # C4: ten training steps of the proposal, forward, backward and update
        dict(name="train_l96_8192", path="train", batch=8192, steps=10, rows=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["resample", "resample", "filter", "step", "batch", "batch", "train"])
    if path == "resample":
        kind = rng.choice(["systematic", "systematic", "multinomial", "metropolis"])
        n = _log(rng, 16, {"systematic": 1 << 23, "multinomial": 1 << 20, "metropolis": 1 << 19}[kind])
        return dict(path=path, kind=kind, n=n, z=rng.choice([0.0, 0.5, 1.0, 2.0, 4.0]),
                    B=rng.randint(8, 32) if kind == "metropolis" else 0, permute=rng.random() < 0.7,
                    offspring=rng.random() < 0.3)
    if path in ("filter", "step"):
        model = rng.choice(["pz", "l96", "l96"])
        dim = 2 if model == "pz" else rng.choice([4, 8, 16, 32, 40, 40])
        prec = "f64" if model == "pz" else rng.choice(["f32", "f32", "f64"])
        kind = rng.choice(["systematic", "systematic", "multinomial", "metropolis"])
        return dict(path=path, model=model, dim=dim, prec=prec, n=_log(rng, 64, 65536),
                    T=_log(rng, 2, 100) if path == "filter" else 1, kind=kind, B=16 if kind == "metropolis" else 0,
                    ess=rng.choice([0.5, 1.0]), paths=path == "filter" and rng.random() < 0.25)
    if path == "batch":
        model, guided = rng.choice(["pz", "l96"]), rng.random() < 0.5
        lo = _log(rng, 100, 2000)
        return dict(path=path, model=model, prec="f64" if model == "pz" else "f32", nf=_log(rng, 2, 128), lo=lo,
                    hi=min(32768, _log(rng, lo, 16 * lo)), T=_log(rng, 2, 30), ess=rng.choice([0.5, 1.0]),
                    kind=rng.choice(["systematic", "mixed"]), guided=guided)
    return dict(path=path, batch=_log(rng, 128, 8192), steps=rng.randint(2, 12), rows=_log(rng, 8192, 65536))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed, tag=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((seed * 1000003 + tag) % (1 << 62))
    return g


def _l96_day(x, F, T=L96_DT, h=L96_H):
    """Lorenz-96 over T by RK4, torch or numpy, components last."""
    roll = torch.roll if isinstance(x, torch.Tensor) else (lambda v, k, a: np.roll(v, k, a))

    def f(v):
        return (roll(v, -1, -1) - roll(v, 2, -1)) * roll(v, 1, -1) - v + F

    for _ in range(int(round(T / h))):
        k1 = f(x)
        k2 = f(x + 0.5 * h * k1)
        k3 = f(x + 0.5 * h * k2)
        x = x + (h / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + f(x + h * k3))
    return x


def _l96_obs(rng, Fs, dim, T):
    """Observations (T, len(Fs), dim) of one run of the model per forcing."""
    F = np.asarray(Fs, float)[:, None]
    x = F + 0.01 * rng.standard_normal((len(Fs), dim))
    y = np.zeros((T, len(Fs), dim))
    for k in range(T):
        x = _l96_day(x, F) + SIGMA_ETA * rng.standard_normal(x.shape)
        y[k] = x + SIGMA_Y * rng.standard_normal(x.shape)
    return y


def _pz_obs(rng, T, m):
    """Daily observations of log P of one run of the plankton model."""
    P, Z = np.exp(math.log(2.0) + 0.2 * rng.standard_normal(2))
    y = np.zeros(T)
    for k in range(T):
        al = math.exp(m.mu + m.sigma * rng.standard_normal())
        for _ in range(100):
            dP, dZ = al * P - m.c * P * Z, m.e * m.c * P * Z - m.m * Z - m.q * Z * Z
            P, Z = P + 0.01 * dP, Z + 0.01 * dZ
        y[k] = math.log(P) + m.sigma_y * rng.standard_normal()
    return y


def _models(case, seed):
    """The models of a case's filters, their sizes, resamplers and seeds."""
    rng = np.random.default_rng([seed, 1])
    if case["path"] != "batch":
        m = ModelPZ() if case["model"] == "pz" else ModelL96(dim=case["dim"], F=L96_F, precision=case["prec"])
        return [m], [case["n"]], [case["kind"]], [seed]
    nf = case["nf"]
    # sizes of the case itself, not of the seed: evenly spread over log N
    q = (np.arange(nf) + 0.5) / nf
    ns = np.floor(np.exp(math.log(case["lo"]) + q * math.log(case["hi"] / case["lo"]))).astype(int)
    ns = [int(n) for n in np.random.default_rng(7).permutation(ns)]
    kinds = [("multinomial" if case["kind"] == "mixed" and f % 2 else "systematic") for f in range(nf)]
    if case["model"] == "l96":
        Fs = np.full(nf, L96_F) if case["guided"] else rng.uniform(6.0, 10.0, nf)
        models = [ModelL96(dim=40, F=float(F), precision=case["prec"]) for F in Fs]
    else:  # chains around the truth, as the posterior holds them
        th = np.array([0.25, 0.3, 0.1, 0.1]) * np.exp(0.1 * rng.standard_normal((nf, 4)))
        models = [ModelPZ(c=float(t[0]), e=float(t[1]), m=float(t[2]), q=float(t[3])) for t in th]
    return models, ns, kinds, [1000 * seed + f for f in range(nf)]


def _observations(case, seed, models):
    rng = np.random.default_rng([seed, 2])
    if case["model"] == "pz":
        y = _pz_obs(rng, case["T"], ModelPZ())
        return np.repeat(y[:, None, None], len(models), 1)  # every chain the same data
    return _l96_obs(rng, [m.F for m in models], models[0].dim, case["T"]).astype(models[0].np_dtype)


def _net_params(rng, din, dout, log_s, w3):
    """A network of the proposal's layout: He-uniform hidden layers and a
    small output layer around (0, log_s)."""
    a1, a2 = math.sqrt(6.0 / din), math.sqrt(6.0 / HIDDEN)
    parts = [a1 * rng.uniform(-1, 1, HIDDEN * din), np.zeros(HIDDEN), a2 * rng.uniform(-1, 1, HIDDEN * HIDDEN),
             0.01 * rng.standard_normal(HIDDEN), w3 * rng.standard_normal(dout * HIDDEN),
             np.concatenate([np.zeros(dout // 2), np.full(dout // 2, log_s)])]
    return np.concatenate(parts).astype(np.float32)


def _proposal(case, seed):
    """The proposal a guided batch keeps: weights and input standardisation
    as training leaves them."""
    rng = np.random.default_rng([seed, 3])
    if case["model"] == "l96":
        p = LearnedProposal(ModelL96(dim=40), L96_DT, 8192, seed)
        p.set_params(_net_params(rng, 80, 80, math.log(SIGMA_ETA), 0.002),
                     np.concatenate([np.full(40, 2.3), np.zeros(40)]),
                     np.concatenate([np.full(40, 1 / 3.6), np.full(40, 1.0)]))
    else:
        p = LearnedProposal(ModelPZ(), 1.0, 8192, seed)
        p.set_params(_net_params(rng, 3, 2, math.log(0.2), 0.005), np.array([0.7, 0.5, 0.0]),
                     np.array([2.0, 2.0, 4.0]))
    return p


def _train_data(case, seed):
    """Triples from the attractor: x_t, one step on, its observation."""
    g = _gen(seed, 4)
    rows = case["rows"]
    x = L96_F + torch.randn((rows, 40), dtype=torch.float64, device=DEV, generator=g)
    for _ in range(40):
        x = _l96_day(x, L96_F)
    xt = x.float()
    m = _l96_day(xt.double(), L96_F)
    xt1 = (m + SIGMA_ETA * torch.randn((rows, 40), dtype=torch.float64, device=DEV, generator=g)).float()
    yt1 = (xt1 + SIGMA_Y * torch.randn((rows, 40), dtype=torch.float32, device=DEV, generator=g)).contiguous()
    P = _net_params(np.random.default_rng([seed, 5]), 80, 80, math.log(SIGMA_ETA), 0.002)
    return xt.contiguous(), xt1.contiguous(), yt1, P


def _log_weights(case, seed):
    """The resampler harness's log-weights and the caller's uniforms."""
    g = _gen(seed, 6)
    x = torch.randn(case["n"], dtype=torch.float64, device=DEV, generator=g) + 0.5 * case["z"]
    u = torch.rand(1, dtype=torch.float64, device=DEV, generator=g) if case["kind"] == "systematic" else None
    return -0.5 * x * x - 0.5 * math.log(2.0 * math.pi), u


def prepare(case, seed):
    path = case["path"]
    if path == "resample":
        lw, u = _log_weights(case, seed)
        return dict(case=case, lw=lw, u=u, r=RESAMPLERS[case["kind"]](max_n=case["n"], B=case["B"]))
    if path == "train":
        xt, xt1, yt1, P = _train_data(case, seed)
        p = LearnedProposal(ModelL96(dim=40), L96_DT, 8192, seed)
        p.set_data(xt, xt1, yt1)
        p.set_params(P)
        return dict(case=case, p=p)
    models, ns, kinds, seeds = _models(case, seed)
    y = _observations(case, seed, models)
    if path in ("filter", "step"):
        pf = BootstrapPF(models[0], ns[0], kinds[0], case["ess"], seeds[0], case["B"])
        if case["paths"]:
            pf.path_cache(case["T"])
        return dict(case=case, pf=pf, y=np.ascontiguousarray(y[:, 0]))
    b = BatchedBootstrapPF(models, ns, kinds, seeds, case["ess"])
    p = None
    if case["guided"]:
        p = _proposal(case, seed)
        b.set_proposal(p)
    _, _, _, offs = b.state()
    cols = torch.cat([torch.arange(o, o + n, device=DEV) for o, n in zip(offs.tolist(), ns)])
    return dict(case=case, b=b, p=p, y=y, cols=cols)


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _dt(case):
    return 1.0 if case["model"] == "pz" else L96_DT


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "resample":
        ess, lW = state["r"].reduce(state["lw"])
        a = state["r"].ancestors(state["lw"], state["u"], permute=case["permute"], with_offspring=case["offspring"])
        return dict(ess=ess, lW=lW, ancestors=a)
    if path == "train":
        trace = state["p"].train(case["steps"], case["batch"], 1e-3)
        return dict(loss=trace, params=state["p"].params()[0])
    if path == "filter":
        pf, n = state["pf"], case["n"]
        ll, inc, ess = pf.filter(state["y"], 0.0, _dt(case))
        x, lw, _ = pf.state()
        # views of the filter's own buffers, valid until its next step: a
        # program that keeps the particles copies them
        out = dict(ll=ll, inc=inc, ess=ess, x=x[:, :n].clone(), lw=lw.clone())
        if case["paths"]:
            out["particle"], out["sampled"] = pf.sample_path()
        return out
    if path == "step":
        pf, n, dt = state["pf"], case["n"], _dt(case)
        pf.init()
        inc, ess = [], []
        for k in range(case["T"]):
            r = pf.step(k * dt, (k + 1) * dt, state["y"][k])
            inc.append(r.log_increment)
            ess.append(r.ess)
        x, lw, _ = pf.state()
        return dict(inc=inc, ess=ess, x=x[:, :n].clone(), lw=lw.clone())
    ll, inc, ess, _ = state["b"].filter(state["y"], 0.0, _dt(case))
    x, lw, _, _ = state["b"].state()
    return dict(ll=ll, inc=inc, ess=ess, x=x[:, state["cols"]], lw=lw[state["cols"]])


def work(case):
    path = case["path"]
    if path == "resample":
        n = case["n"]
        draws = n * case["B"] if case["kind"] == "metropolis" else n if case["kind"] == "multinomial" else 0
        return dict(bytes=8 * n + 4 * n * (2 if case["offspring"] else 1), flops=40 * n + 60 * draws)
    if path == "train":
        B = case["batch"]
        weights = 80 * HIDDEN + HIDDEN * HIDDEN + HIDDEN * 80
        return dict(bytes=case["steps"] * (B * 4 * 160 + 24 * weights), flops=case["steps"] * 6 * B * weights)
    if path == "batch":
        # the sizes of _models, without the seed
        nf = case["nf"]
        total = sum(math.floor(math.exp(math.log(case["lo"]) + (f + 0.5) / nf * math.log(case["hi"] / case["lo"])))
                    for f in range(nf))
        dim = 2 if case["model"] == "pz" else 40
    else:
        total, dim = case["n"], case["dim"]
    size = 4 if case["prec"] == "f32" else 8
    # state and log-weight in and out; RK4: 5 sub-steps of 34 operations a
    # component, noise and density; RK4(3): about 8 sub-steps of 130
    flops = 8 * 130 + 100 if case["model"] == "pz" else dim * (34 * 5 + 40)
    if case.get("guided"):
        flops += 2 * (80 * HIDDEN + HIDDEN * HIDDEN + HIDDEN * 80 if case["model"] == "l96" else HIDDEN * (HIDDEN + 5))
    return dict(bytes=case["T"] * total * (2 * dim * size + 16), flops=case["T"] * total * flops)


# --------------------------------------------------------------------------
# the same in 64 bits, plain torch
# --------------------------------------------------------------------------
M32 = 0xFFFFFFFF
NOISE, INIT, SYSTEMATIC, DATA = 0, 1, 2, 5  # the random stream's tags


def _philox(seed, c0, c1, c2, c3):
    """Philox4x32-10 (Salmon et al. 2011) of tensor counters c0 under the key
    `seed` (a tensor of c0's shape or a number); four int64 tensors."""
    c = [c0, torch.full_like(c0, c1), torch.full_like(c0, c2), torch.full_like(c0, c3)]
    key = seed if isinstance(seed, torch.Tensor) else torch.full_like(c0, seed)
    k0, k1 = key & M32, (key >> 32) & M32
    for _ in range(10):
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((b >> 32) & M32) ^ c[1] ^ k0, b & M32, ((a >> 32) & M32) ^ c[3] ^ k1, a & M32]
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    return c


def _normals(r0, r1):
    ua = (2.0 * (r0 >> 9).double() + 1.0) * 2.0 ** -24
    ub = (2.0 * (r1 >> 9).double() + 1.0) * 2.0 ** -24
    r = torch.sqrt(-2.0 * torch.log(ua))
    return r * torch.cos(2.0 * math.pi * ub), r * torch.sin(2.0 * math.pi * ub)


def _normals4(seed, p, step, dim, tag):
    z = []
    for b in range((dim + 3) // 4):
        r = _philox(seed, p, step, b, tag)
        z += [*_normals(r[0], r[1]), *_normals(r[2], r[3])]
    return torch.stack(z[:dim], -1)


def _pz_day(P, Z, al, th, t1, t2):
    """The adaptive RK4(3)5[2R+]C of Kennedy, Carpenter & Lewis (2000) with the
    model's step control; every argument a tensor but the times."""
    A = (0.225022458725713, 0.544043312951405, 0.144568243493995, 0.786664342198357)
    Bc = (0.0512293066403392, 0.380954825726402, -0.373352596392383, 0.592501285026362, 0.34866717899928)
    E = (-0.0859880154628801, 0.189074063397015, -0.144145875232852, -0.0317933915175331, 0.0728532188162504)
    cc, ee, mm, qq = th

    def f(P, Z):
        return al * P - cc * P * Z, ee * cc * P * Z - mm * Z - qq * Z * Z

    t, h = torch.full_like(P, t1), torch.full_like(P, 0.1)
    old, lfo = [P, Z], torch.full_like(P, math.log(1e-4))
    x = [P, Z]
    beta, logsafe = 0.04, math.log(0.9)
    expo = 0.5 * (0.2 - 0.04 * 0.75)
    while bool((t < t2).any()):
        go = t < t2
        h = torch.where(go & (1.01 * h + t - t2 > 0), t2 - t, h)
        r1, err, S = list(x), [0.0, 0.0], list(x)
        r2 = None
        for s in range(5):
            k = f(*S)
            err = [a + E[s] * b for a, b in zip(err, k)]
            if s == 4:
                r1 = [a + Bc[4] * h * b for a, b in zip(r1, k)]
            elif s % 2 == 0:
                r1 = [a + A[s] * h * b for a, b in zip(r1, k)]
                r2 = [a + (Bc[s] - A[s]) * h * b for a, b in zip(r1, k)]
                S = r1
            else:
                r2 = [a + A[s] * h * b for a, b in zip(r2, k)]
                r1 = [a + (Bc[s] - A[s]) * h * b for a, b in zip(r2, k)]
                S = r2
        rel = [(a * h) / (1e-3 + 1e-3 * torch.maximum(o.abs(), b.abs())) for a, o, b in zip(err, old, r1)]
        e2 = (rel[0] ** 2 + rel[1] ** 2) / 2.0
        good = go & (e2 <= 1.0)
        bad = go & ~good
        t = torch.where(good, t + h, t)
        x = [torch.where(good, b, a) for a, b in zip(x, r1)]
        more = t < t2
        old = [torch.where(good & more, b, a) for a, b in zip(old, r1)]
        lf = expo * torch.log(e2)
        up = torch.exp(beta * lfo + logsafe - lf).clamp(0.2, 10.0)
        down = torch.exp(logsafe - lf).clamp(min=0.2)
        h = torch.where(good & more, h * up, torch.where(bad, h * down, h))
        lfo = torch.where(good & more, 0.5 * torch.log(e2.clamp(min=1e-8)), lfo)
    return x


def _exact_pz(case, seed):
    models, ns, kinds, seeds = _models(case, seed)
    y = _observations(case, seed, models)
    p = torch.cat([torch.arange(n, device=DEV) for n in ns])
    key = torch.cat([torch.full((n,), s, device=DEV) for n, s in zip(ns, seeds)])
    th = [torch.cat([torch.full((n,), getattr(m, k), dtype=torch.float64, device=DEV) for n, m in zip(ns, models)])
          for k in ("c", "e", "m", "q")]
    ends = np.cumsum([0] + ns)
    r = _philox(key, p, 0, 0, INIT)
    z0, z1 = _normals(r[0], r[1])
    P, Z = torch.exp(math.log(2.0) + 0.2 * z0), torch.exp(math.log(2.0) + 0.2 * z1)
    lw = torch.zeros_like(P)
    m0, T, F = ModelPZ(), case["T"], len(ns)
    ll, again = np.zeros(F), [False] * F
    inc, ess = np.zeros((T, F)), np.zeros((T, F))
    for k in range(1, T + 1):
        src = torch.arange(P.numel(), device=DEV)
        for f in range(F):
            if not again[f]:
                continue
            s, n = slice(ends[f], ends[f + 1]), ns[f]
            W = torch.cumsum(torch.exp(lw[s] - lw[s].max()), 0)
            u = _philox(seeds[f], torch.zeros(1, dtype=torch.int64, device=DEV), k, 0, SYSTEMATIC)
            a = (2.0 * (((u[0] << 20) | (u[1] >> 12))).double() + 1.0) * 2.0 ** -53
            Os = (W / W[-1] * n + a).long().clamp(max=n)
            o = torch.diff(Os, prepend=Os.new_zeros(1))
            extra = torch.repeat_interleave(torch.arange(n, device=DEV), (o - 1).clamp(min=0))
            free = torch.nonzero(o == 0).flatten()
            src[ends[f] + free] = ends[f] + extra[:free.numel()]
            lw[s] = ll[f]
        P, Z = P[src], Z[src]
        r = _philox(key, p, k, 0, NOISE)
        al = torch.exp(m0.mu + m0.sigma * _normals(r[0], r[1])[0])
        P, Z = _pz_day(P, Z, al, th, (k - 1.0), float(k))
        lw = lw - 0.5 * ((float(y[k - 1, 0, 0]) - torch.log(P)) / m0.sigma_y) ** 2 - 0.5 * math.log(2 * math.pi) \
            - math.log(m0.sigma_y)
        for f in range(F):
            l = lw[ends[f]:ends[f + 1]]
            mx = l.max()
            e = torch.exp(l - mx)
            s1, s2, mx = torch.stack([e.sum(), (e * e).sum(), mx]).tolist()
            lW = mx + math.log(s1) - math.log(ns[f])
            inc[k - 1, f], ess[k - 1, f] = lW - ll[f], s1 * s1 / s2
            ll[f] = lW
            again[f] = ess[k - 1, f] < case["ess"] * ns[f]
    out = dict(ll=ll, inc=inc, ess=ess, x=torch.stack([P, Z]), lw=lw)
    if case["path"] != "batch":
        out.update(ll=float(ll[0]), inc=inc[:, 0], ess=ess[:, 0])
    if case["path"] == "step":
        out = dict(inc=inc[:, 0].tolist(), ess=ess[:, 0].tolist(), x=out["x"], lw=lw)
    return out


def _exact_l96_step(case, seed):
    models, ns, _, seeds = _models(case, seed)
    m, n, D = models[0], ns[0], models[0].dim
    y = torch.from_numpy(_observations(case, seed, models)[0, 0].astype(float)).to(DEV)
    p = torch.arange(n, device=DEV)
    x = L96_F + m.x0_std * _normals4(seeds[0], p, 0, D, INIT)
    x = _l96_day(x, L96_F) + SIGMA_ETA * _normals4(seeds[0], p, 1, D, NOISE)
    lw = (-0.5 * ((y - x) / SIGMA_Y) ** 2 - 0.5 * math.log(2 * math.pi) - math.log(SIGMA_Y)).sum(-1)
    e = torch.exp(lw - lw.max())
    ess, ll = float(e.sum() ** 2 / (e * e).sum()), float(torch.logsumexp(lw, 0)) - math.log(n)
    return dict(inc=[ll], ess=[ess], x=x.t().contiguous(), lw=lw)


def _exact_train(case, seed):
    xt, xt1, yt1, flat = _train_data(case, seed)
    n, B, steps = case["rows"], case["batch"], case["steps"]
    xt, xt1, yt1 = xt.double(), xt1.double(), yt1.double()
    m = _l96_day(xt, L96_F)
    u = torch.cat([xt, yt1 - m], 1)
    head = u[:65536]
    u = (u - head.mean(0)) / head.var(0, unbiased=False).sqrt()
    r0 = xt1 - m
    P = torch.from_numpy(flat).double().to(DEV).requires_grad_()
    sizes = [HIDDEN * 80, HIDDEN, HIDDEN * HIDDEN, HIDDEN, 80 * HIDDEN, 80]
    m1, m2 = torch.zeros_like(P), torch.zeros_like(P)
    loss = np.zeros(steps, np.float64)
    warm = max(steps // 20, 1)
    for s in range(steps):
        w = [v.cpu().numpy().astype(np.uint64) for v in _philox(seed, torch.arange(B, device=DEV), s, 0, DATA)[:2]]
        rows = torch.from_numpy((((w[0] << np.uint64(32)) | w[1]) % np.uint64(n)).astype(np.int64)).to(DEV)
        W1, b1, W2, b2, W3, b3 = torch.split(P, sizes)
        h = torch.relu(u[rows] @ W1.view(HIDDEN, 80).t() + b1)
        h = torch.relu(h @ W2.view(HIDDEN, HIDDEN).t() + b2)
        o = h @ W3.view(80, HIDDEN).t() + b3
        sc = o[:, 40:].clamp(-7.0, 3.0)
        l = (sc + 0.5 * (r0[rows] - o[:, :40]) ** 2 * torch.exp(-2.0 * sc)).sum(1).mean()
        (g,) = torch.autograd.grad(l, P)
        loss[s] = float(l)
        lr = 1e-3 * min(1.0, (s + 1) / warm) * (0.1 + 0.45 * (1.0 + math.cos(math.pi * s / steps)))
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        step = lr * (m1 / (1 - 0.9 ** (s + 1))) / ((m2 / (1 - 0.999 ** (s + 1))).sqrt() + 1e-8)
        P = (P.detach() - step).requires_grad_()
    return dict(loss=loss, params=P.detach().cpu().numpy())


def exact(case, seed):
    path = case["path"]
    if path == "resample":
        lw = _log_weights(case, seed)[0].cpu().numpy()
        mx = lw.max()
        e = np.exp(lw - mx)
        s1, s2 = math.fsum(e), math.fsum(e * e)
        return dict(ess=s1 * s1 / s2, lW=float(mx) + math.log(s1) - math.log(case["n"]), ancestors=None)
    if path == "train":
        return _exact_train(case, seed)
    if path == "step" and case["model"] == "l96" and case["T"] == 1:
        return _exact_l96_step(case, seed)
    if case["model"] == "pz" and not case.get("guided") and case["kind"] == "systematic" and not case.get("paths"):
        return _exact_pz(case, seed)
    # Lorenz-96 is chaotic and resampling discontinuous: over several steps
    # the 32-bit and BF16 filters have no 64-bit counterpart, particle by
    # particle; nor have the other resamplers' ancestors without their draws
    return None
