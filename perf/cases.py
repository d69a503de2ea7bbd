"""Timing cases of the CATMIP path through its public entry points.

``listed()`` names the cases; each is a dict of plain values.  ``prepare(case, seed)`` builds
what a program holds before the call (model, observations, samples, buffers), ``run(state)``
makes one pass and returns its outputs, ``work(case)`` says what the pass cannot do without and
``exact(case, seed)`` computes the same outputs in 64 bits with torch or numpy alone, where that
takes seconds.  ``draw(rng)`` gives further cases of the same ranges.
"""
import math

import numpy as np
import torch

from altar_gb300 import Application
from altar_gb300.autotune import tune
from altar_gb300.bayesian import COV, Annealer, Brent, CoolingStep, Grid, Surrogate
from altar_gb300.distributions import Uniform
from altar_gb300.models import CDM, Contiguous, DenseMogi, Linear, Mogi, Reverso
from altar_gb300.models.observations import Observations
from altar_gb300.models.reverso import PSETS
from altar_gb300.simulations import RNG, Job

DEV = "cuda"
NU = 0.25
LOS = ((0.38, -0.08, 0.92), (-0.61, 0.11, 0.78), (0.09, 0.56, 0.82))     # one per dataset
# x, y, depth, opening, semi-axes, rotations (degrees)
CDM_PRIORS = [(-1e4, 1e4)] * 2 + [(1e3, 1e4), (-50.0, 50.0)] + [(100.0, 3000.0)] * 3 + [(-90.0, 90.0)] * 3
MOGI_PRIORS = [(-1e4, 1e4)] * 2 + [(1e3, 8e3), (5.0, 7.0)]               # x, y, depth, log10 ΔV
REVERSO_PRIORS = [(0.4, 0.8), (2500.0, 3500.0), (3500.0, 4500.0), (1500.0, 2500.0), (1500.0, 2500.0), (1.0, 2.0)]
REVERSO = dict(v=0.25, mu=2000.0, drho=300.0, G=20.0e9, g=9.81)
YEAR = 365.25 * 24 * 3600


def listed():
    return [
        # the CDM workload's population at one Metropolis step: 200 x 200 InSAR grid, launch
        # shape from the autotuner as the quick start has it
        dict(name="cdm_population", kind="cdm", chains=32768, stations=40000, grid=True, datasets=0, spread=1.0,
             call="hook", tuned=True),
        # the exact fields of the 256 check chains that delayed acceptance looks at in each stage
        dict(name="cdm_check_fields", kind="cdm", chains=256, stations=40000, grid=True, datasets=0, spread=0.05,
             call="residuals", tuned=False),
        # a small campaign: two scattered datasets with an offset each, the walk's call (mask, early rejection)
        dict(name="cdm_campaign", kind="cdm", chains=1999, stations=577, grid=False, datasets=2, spread=0.3,
             call="walk", tuned=False),
        # a Mogi population on three scattered datasets with offsets, log10 ΔV as in the reference
        dict(name="mogi_population", kind="mogi", chains=16384, stations=10007, datasets=3),
        # two Mogi sources, three datasets of uneven size with dense Cd (a tenth of the batched workload's sizes)
        dict(name="dense_mogi", kind="dense", chains=16384, m0=1200, m1=3000, m2=750),
        # the linear workload at its own size, on the tensor cores
        dict(name="linear_tensor", kind="linear", chains=16384, obs=4096, params=256, tensor=True),
        # a small linear model evaluated in FP64, the precision option
        dict(name="linear_fp64", kind="linear", chains=2003, obs=997, params=61, tensor=False),
        # one stage's schedule for the CDM population: β by the grid solver, Σ, resampling
        dict(name="cov_stage", kind="cov", chains=32768, params=10, scale=3e4, solver="grid"),
        # whole runs from the prior to β = 1: the reference's Reverso example, and plain CATMIP on one Mogi source
        dict(name="reverso_anneal", kind="anneal", model="reverso", chains=4096, obs=35, steps=20),
        dict(name="mogi_anneal", kind="anneal", model="mogi", chains=1024, obs=1024, steps=5),
        # the surrogate of delayed acceptance: prediction for a population, one training epoch
        dict(name="surrogate_predict", kind="predict", chains=32768),
        dict(name="surrogate_epoch", kind="train", samples=4096, batch=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cdm", "cdm", "mogi", "dense", "linear", "cov", "anneal", "predict", "train"])
    if kind == "cdm":
        n = _log_int(rng, 32, 32768)
        m = _log_int(rng, 64, min(40000, 1.2e9 / n))
        return dict(kind=kind, chains=n, stations=m, grid=rng.random() < 0.5, datasets=rng.choice([0, 1, 3]),
                    spread=math.exp(rng.uniform(math.log(0.03), 0.0)),
                    call=rng.choice(["hook", "residuals", "walk"] if n * m < 4e7 else ["hook", "walk"]), tuned=False)
    if kind == "mogi":
        n = _log_int(rng, 64, 32768)
        return dict(kind=kind, chains=n, stations=_log_int(rng, 64, min(40000, 4e8 / n)), datasets=rng.choice([0, 2]))
    if kind == "dense":
        return dict(kind=kind, chains=_log_int(rng, 256, 16384), m0=_log_int(rng, 100, 1300),
                    m1=_log_int(rng, 300, 3000), m2=_log_int(rng, 60, 800))
    if kind == "linear":
        tensor = rng.random() < 0.7
        if tensor:
            return dict(kind=kind, chains=_log_int(rng, 128, 16384), obs=_log_int(rng, 100, 4096),
                        params=_log_int(rng, 8, 256), tensor=True)
        return dict(kind=kind, chains=_log_int(rng, 64, 4096), obs=_log_int(rng, 50, 1500),
                    params=_log_int(rng, 4, 128), tensor=False)
    if kind == "cov":
        return dict(kind=kind, chains=_log_int(rng, 256, 65536), params=rng.randint(4, 24),
                    scale=math.exp(rng.uniform(math.log(2.0), math.log(1e6))), solver=rng.choice(["grid", "grid", "brent"]))
    if kind == "anneal":
        if rng.random() < 0.5:
            return dict(kind=kind, model="reverso", chains=_log_int(rng, 512, 4096), obs=_log_int(rng, 10, 120),
                        steps=rng.randint(4, 20))
        return dict(kind=kind, model="mogi", chains=_log_int(rng, 256, 4096), obs=_log_int(rng, 100, 4000),
                    steps=rng.randint(3, 10))
    if kind == "predict":
        return dict(kind=kind, chains=_log_int(rng, 256, 65536))
    return dict(kind=kind, samples=_log_int(rng, 1024, 8192), batch=rng.choice([512, 1024, 2048]))


# ---------------------------------------------------------------------------
# inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 62))


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _below(theta):
    """CDM sources whose three rectangles all lie under the surface."""
    om = torch.deg2rad(theta[:, 7:10])
    s, c = torch.sin(om), torch.cos(om)
    up = torch.stack([s[:, 1], -c[:, 1] * s[:, 0], c[:, 1] * c[:, 0]], 1).abs() * theta[:, 4:7]
    top = torch.maximum(torch.maximum(up[:, 0] + up[:, 1], up[:, 0] + up[:, 2]), up[:, 1] + up[:, 2])
    return theta[:, 2] > top


def _cdm_sources(g, n, spread, truth=None):
    """Sources under the surface: prior draws, or draws around `truth` as wide as `spread` of the prior."""
    lo, hi = (torch.tensor(v, dtype=torch.float64, device=DEV) for v in zip(*CDM_PRIORS))
    rows = []
    while sum(r.shape[0] for r in rows) < n:
        u = torch.rand(2 * n + 64, 10, generator=g, device=DEV, dtype=torch.float64)
        th = lo + u * (hi - lo) if truth is None or spread >= 1.0 else truth + (u - 0.5) * spread * (hi - lo)
        ok = _below(th) & ((th >= lo) & (th <= hi)).all(1)
        rows.append(th[ok])
    return torch.cat(rows)[:n].contiguous()


def _stations(g, m, grid, half=20e3):
    if grid:
        side = int(math.ceil(math.sqrt(m)))
        t = torch.linspace(-half, half, side, dtype=torch.float64, device=DEV)
        y, x = torch.meshgrid(t, t, indexing="ij")
        return x.reshape(-1)[:m].contiguous(), y.reshape(-1)[:m].contiguous()
    return _uniform(g, (m,), -half, half), _uniform(g, (m,), -half, half)


def _datasets(m, k):
    """Dataset of each station and its line of sight (k = 0: one dataset without an offset parameter)."""
    oid = (torch.arange(m, device=DEV) * max(k, 1)) // m
    return oid, torch.tensor(LOS, dtype=torch.float64, device=DEV)[oid]


def _cdm_inputs(case, seed):
    g = _gen(seed)
    n, m, k = case["chains"], case["stations"], case["datasets"]
    x, y = _stations(g, m, case["grid"])
    oid, los = _datasets(m, k)
    truth = _cdm_sources(g, 1, 1.0)
    theta = _cdm_sources(g, n, case["spread"], truth)
    now = _cdm_sources(g, n, case["spread"], truth) if case["call"] == "walk" else None
    off = 0.01 * _normal(g, n, k) if k else None
    shift = 0.01 * _normal(g, k)[oid] if k else 0.0
    d = _cdm_los(truth, x, y, los)[0] + shift + 3e-3 * _normal(g, m)
    if k:
        theta = torch.cat([theta, off], 1).contiguous()
    inp = dict(x=x, y=y, los=los, d=d, oid=oid, theta=theta, var=9e-6)
    if now is not None:
        # the current states' log-likelihoods and the accept test's uniforms give each proposal its floor;
        # one proposal in twenty has left the prior's support, one in thirty rises above the surface
        if k:
            now = torch.cat([now, off], 1)
        beta = 1e-3
        inp["floor"] = _cdm_llk(inp, now)[0] + torch.log(torch.rand(n, generator=g, device=DEV, dtype=torch.float64)) / beta
        inp["mask"] = (torch.rand(n, generator=g, device=DEV) < 0.05).to(torch.int32)
        high = torch.rand(n, generator=g, device=DEV) < 1 / 30
        theta[high, 2] *= 0.05
    return inp


def _psets(names, counts, bounds, k=0):
    psets = {nm: Contiguous(c, Uniform(b)) for nm, c, b in zip(names, counts, bounds)}
    if k:
        psets["offsets"] = Contiguous(k, Uniform((-1.0, 1.0)))
    return psets


def _cdm_psets(k):
    return _psets(["location", "depth", "opening", "a", "omega"], [2, 1, 1, 3, 3],
                  [CDM_PRIORS[j] for j in (0, 2, 3, 4, 7)], k)


def _observations(inp, k):
    cpu = lambda t: t.cpu().numpy()                             # noqa: E731
    return Observations(cpu(inp["x"]), cpu(inp["y"]), cpu(inp["los"]), cpu(inp["d"]), inp["var"],
                        oid=cpu(inp["oid"]) if k else None)


def _ready(model, chains, seed, steps=5, controller=None):
    return Application(model, job=Job(chains=max(2, chains), steps=steps), rng=RNG(seed), controller=controller).initialize()


def _step(theta):
    n = theta.shape[0]
    zeros = lambda: torch.zeros(n, dtype=torch.float64, device=DEV)      # noqa: E731
    return CoolingStep(beta=0.0, theta=theta, likelihoods=(zeros(), zeros(), zeros()))


def _mogi_inputs(case, seed):
    g = _gen(seed)
    n, m, k = case["chains"], case["stations"], case["datasets"]
    x, y = _stations(g, m, False, 25e3)
    oid, los = _datasets(m, k)
    lo, hi = (torch.tensor(v, dtype=torch.float64, device=DEV) for v in zip(*MOGI_PRIORS))
    rows = lo + torch.rand(n + 1, 4, generator=g, device=DEV, dtype=torch.float64) * (hi - lo)
    d = _mogi_los(rows[:1], x, y, los)[0] + 5e-3 * _normal(g, m)
    theta = rows[1:]
    if k:
        theta = torch.cat([theta, 0.01 * _normal(g, n, k)], 1)
    return dict(x=x, y=y, los=los, d=d, oid=oid, theta=theta.contiguous(), var=2.5e-5)


def _dense_inputs(case, seed):
    g = _gen(seed)
    truth = torch.tensor([[-4e3, 1e3, 3e3, 6.3, 3e3, -2e3, 4e3, 6.1]], dtype=torch.float64, device=DEV)
    sets = []
    for m, los in zip((case["m0"], case["m1"], case["m2"]), LOS):
        x, y = _stations(g, m, False, 25e3)
        cd = 1.6e-5 * torch.exp(-torch.hypot(x[:, None] - x, y[:, None] - y) / 2e3)
        cd += 1e-9 * torch.eye(m, dtype=torch.float64, device=DEV)
        lv = torch.tensor([los], dtype=torch.float64, device=DEV).expand(m, 3)
        d = _mogi_los(truth, x, y, lv, 2)[0] + torch.linalg.cholesky(cd) @ _normal(g, m)
        sets.append(dict(x=x, y=y, los=lv, d=d, cd=cd))
    wide = torch.tensor([500.0, 500.0, 300.0, 0.05] * 2, dtype=torch.float64, device=DEV)
    theta = truth + _normal(g, case["chains"], 8) * wide
    return sets, theta.contiguous()


def _linear_inputs(case, seed):
    g = _gen(seed)
    m, p = case["obs"], case["params"]
    G = _normal(g, m, p)
    x, y = _stations(g, m, False, 25e3)
    cd = 1e-4 * torch.exp(-torch.hypot(x[:, None] - x, y[:, None] - y) / 2e3)
    truth = _uniform(g, (p,), -1.0, 1.0)
    d = G @ truth + torch.linalg.cholesky(cd) @ _normal(g, m)
    return G, d, cd, _uniform(g, (case["chains"], p), -1.0, 1.0)


def _cov_inputs(case, seed):
    """A population and its data log-likelihoods: minus a quadratic form of θ, `scale` times a χ² in size."""
    g = _gen(seed)
    n, p = case["chains"], case["params"]
    z = _normal(g, n, p)
    mix = torch.eye(p, dtype=torch.float64, device=DEV) + 0.3 * _normal(g, p, p) / math.sqrt(p)
    theta = (z @ mix) * torch.logspace(0, 3, p, dtype=torch.float64, device=DEV) + 50.0
    data = -0.5 * case["scale"] * (z * z * torch.linspace(0.2, 1.0, p, dtype=torch.float64, device=DEV)).sum(1) - 2e3
    return theta.contiguous(), torch.full((n,), -30.0, dtype=torch.float64, device=DEV), data


def _reverso_points(k):
    """k observation points: times spread over 10^-6 .. 1 year, 1 to 5 km east."""
    i = np.arange(k)
    return np.stack([10.0 ** (-6.0 + 6.0 * (i // 5) / max(1, (k - 1) // 5)) * YEAR, 1000.0 * (1 + i % 5), 0.0 * i], 1)


def _network(seed):
    rng = np.random.default_rng(seed)
    sizes = Surrogate().sizes
    flat = []
    for fi, fo in zip(sizes[:-1], sizes[1:]):
        flat += [rng.normal(0.0, math.sqrt(2.0 / fi), fo * fi), rng.normal(0.0, 0.05, fo)]
    return sizes, np.concatenate(flat).astype(np.float32)


def _fields(g, count, m):
    """Smooth fields of `count` sources on m stations (sums of a few bumps), in metres."""
    x = torch.linspace(-1, 1, m, device=DEV)
    c, w, a = (torch.rand(count, 6, generator=g, device=DEV) for _ in range(3))
    return (0.2 * (a - 0.5)[:, :, None] / (1 + ((x - 2 * c[:, :, None] + 1) / (0.1 + w[:, :, None])) ** 2)).sum(1)


def _predict_inputs(case, seed):
    g = _gen(seed)
    fields = _fields(g, 512, 2048)
    d = fields[0] + 3e-3 * torch.randn(2048, generator=g, device=DEV)
    theta = _uniform(g, (case["chains"], 10), -1.0, 1.0) * 2e3 + 1e3
    lo, hi = torch.full((2, 10), -1e3, dtype=torch.float64, device=DEV)
    return fields, d, theta, lo.contiguous(), (hi + 4e3).contiguous()


def _train_inputs(case, seed):
    g = _gen(seed)
    x = torch.rand(case["samples"], 10, generator=g, device=DEV) * 2 - 1
    mix = torch.randn(10, 64, generator=g, device=DEV) / 3
    return x, torch.sin(2 * x @ mix) + 0.1 * (x @ mix) ** 2


# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "cdm":
        inp = _cdm_inputs(case, seed)
        model = CDM(_cdm_psets(case["datasets"]), observations=_observations(inp, case["datasets"]))
        _ready(model, case["chains"], seed)
        step = _step(inp["theta"])
        if case["tuned"]:
            tune(model.strategy, step.theta, use_cache=False)
        st = dict(case=case, model=model, step=step)
        if case["call"] == "residuals":
            st["residuals"] = torch.zeros(case["chains"], model.strategy.stations.m_padded, device=DEV)
        if case["call"] == "walk":
            st.update(mask=inp["mask"], floor=inp["floor"])
        return st
    if kind == "mogi":
        inp = _mogi_inputs(case, seed)
        psets = _psets(["location", "depth", "source"], [2, 1, 1], [MOGI_PRIORS[j] for j in (0, 2, 3)], case["datasets"])
        model = Mogi(psets, observations=_observations(inp, case["datasets"]))
        _ready(model, case["chains"], seed)
        return dict(case=case, model=model, step=_step(inp["theta"]))
    if kind == "dense":
        sets, theta = _dense_inputs(case, seed)
        data = [{k: (v if k == "cd" else v.cpu().numpy()) for k, v in s.items()} for s in sets]
        psets = {}
        for s in range(2):
            psets.update({f"location{s}": Contiguous(2, Uniform(MOGI_PRIORS[0])),
                          f"depth{s}": Contiguous(1, Uniform(MOGI_PRIORS[2])),
                          f"source{s}": Contiguous(1, Uniform(MOGI_PRIORS[3]))})
        model = DenseMogi(psets, data)
        _ready(model, case["chains"], seed)
        return dict(case=case, model=model, step=_step(theta))
    if kind == "linear":
        G, d, cd, theta = _linear_inputs(case, seed)
        model = Linear({"theta": Contiguous(case["params"], Uniform((-1.0, 1.0)))}, green=G.cpu().numpy(),
                       data=d.cpu().numpy(), cd=cd.cpu().numpy(), tensor_cores=case["tensor"])
        _ready(model, case["chains"], seed)
        return dict(case=case, model=model, step=_step(theta))
    if kind == "cov":
        theta, prior, data = _cov_inputs(case, seed)
        step = CoolingStep(beta=0.0, theta=theta, likelihoods=(prior, data, prior.clone()))
        sched = COV(solver=Brent() if case["solver"] == "brent" else Grid())
        sched.seed = int(seed) & 0xFFFFFFFF
        sched.solver.initialize(application=None, scheduler=sched)
        return dict(case=case, step=step, sched=sched)
    if kind == "anneal":
        rng = np.random.default_rng(seed)
        if case["model"] == "reverso":
            txy = _reverso_points(case["obs"])
            psets = lambda: {nm: Contiguous(1, Uniform(b)) for nm, b in zip(PSETS, REVERSO_PRIORS)}  # noqa: E731
            truth = np.array([[0.6, 3.0e3, 4.0e3, 2.0e3, 2.2e3, 1.5]])
            u = _reverso_fields(truth, txy)[0]
            var = np.maximum(0.05 * u, 0.01) ** 2
            model = Reverso(psets(), txy=txy, d=u + 0.2 * np.sqrt(var) * rng.normal(size=u.shape), var=var, **REVERSO)
        else:
            m = case["obs"]
            side = int(math.ceil(math.sqrt(m)))
            t = np.linspace(-15e3, 15e3, side)
            X, Y = (a.ravel()[:m] for a in np.meshgrid(t, t))
            truth = torch.tensor([[0.0, 0.0, 3e3, math.log10(2e6)]], dtype=torch.float64, device=DEV)
            dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)      # noqa: E731
            u = _mogi_los(truth, dev(X), dev(Y), dev(np.tile(LOS[0], (m, 1))))[0].cpu().numpy()
            psets = _psets(["location", "depth", "source"], [2, 1, 1], [MOGI_PRIORS[0], MOGI_PRIORS[2], (1e5, 1e7)])
            model = Mogi(psets, observations=Observations(X, Y, [LOS[0]], u + rng.normal(0, 5e-3, m), 2.5e-5),
                         log_strength=False)
        return dict(case=case, model=model,
                    app=_ready(model, case["chains"], seed, steps=case["steps"], controller=Annealer()))
    if kind == "predict":
        fields, d, theta, lo, hi = _predict_inputs(case, seed)
        sur = Surrogate().init_params()
        sur.set_params(_network(seed)[1])
        sur.fit_basis(fields, torch.full((2048,), 1 / 9e-6, device=DEV), d, 5e3)
        return dict(case=case, sur=sur, theta=theta, lo=lo, hi=hi, bufs=sur.buffers(*theta.shape),
                    out=torch.zeros(case["chains"], dtype=torch.float64, device=DEV))
    x, y = _train_inputs(case, seed)
    sur = Surrogate(batch=case["batch"]).init_params()
    sur.reserve(case["samples"], 10)
    sur.add(x, y)
    return dict(case=case, sur=sur, flat=torch.from_numpy(_network(seed)[1]).to(DEV))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("cdm", "mogi", "dense", "linear"):
        model, step = state["model"], state["step"]
        if case.get("call") == "residuals":
            model.strategy.forward(step.theta, step.data, residuals=state["residuals"])
            return {"llk": step.data, "residuals": state["residuals"]}
        if case.get("call") == "walk":
            mask = state["mask"]
            model.strategy.forward(step.theta, step.data, mask=mask, status=mask, floor=state["floor"])
            return {"llk": step.data, "mask": mask}
        model.dataLikelihood(step)
        return {"llk": step.data}
    if kind == "cov":
        # the three parts of COV.update, from β = 0 and the same population in each pass
        step, sched = state["step"], state["sched"]
        step.beta = 0.0
        sched.updateTemperature(step)
        sched.computeCovariance(step)
        theta, (prior, data, post) = sched.rank(step)
        s = step.state
        return {"beta": s.beta, "dbeta_cov": s.dbeta_cov, "w": s.w, "sigma": s.sigma, "theta": theta, "prior": prior,
                "data": data, "posterior": post}
    if kind == "anneal":
        state["model"].posterior(state["app"])
        step = state["app"].controller.worker.step
        return {"beta": step.state.beta, "theta": step.theta, "prior": step.prior, "data": step.data,
                "posterior": step.posterior, "sigma": step.sigma}
    if kind == "predict":
        sur = state["sur"]
        sur.predict(state["theta"], state["lo"], state["hi"], state["out"], state["bufs"])
        return {"llk": state["out"], "coefficients": state["bufs"][1]}
    # one epoch from the given weights
    sur = state["sur"]
    sur.set_params(state["flat"])
    sur.m.zero_()
    sur.v.zero_()
    sur.step_count = 0
    sur.losses = []
    sur.train(epochs=1)
    return {"params": sur.params, "m": sur.m, "v": sur.v, "loss": sur.losses[0]}


def work(case):
    kind, n = case["kind"], case.get("chains", 0)
    if kind == "cdm":
        m = case["stations"]
        b = 8 * n * (10 + case["datasets"]) + 40 * m + 8 * n + (4 * n * m if case["call"] == "residuals" else 0)
        # ~1,600 FLOP per pair: far rectangles as point dislocations, near ones by their sides
        return dict(bytes=b, flops=1600.0 * n * m)
    if kind == "mogi":
        m = case["stations"]
        return dict(bytes=8 * n * (4 + case["datasets"]) + 40 * m + 8 * n, flops=41.0 * n * m)
    if kind == "dense":
        ms = (case["m0"], case["m1"], case["m2"])
        # W = L⁻¹ is triangular: m (m + 1) FLOP per chain and dataset
        return dict(bytes=8 * n * 9 + sum(40 * m + 4 * m * m / 2 for m in ms),
                    flops=n * sum(m * (m + 1.0) + 82 * m for m in ms))
    if kind == "linear":
        m, p = case["obs"], case["params"]
        return dict(bytes=8 * (n * p + n) + (4 if case["tensor"] else 8) * m * p, flops=2.0 * n * m * p)
    if kind == "cov":
        p = case["params"]
        return dict(bytes=8 * n * (2 * (p + 2) + 3), flops=n * (60.0 * 20 + p * (p + 3) + p))
    if kind == "anneal":
        per = 180.0 if case["model"] == "reverso" else 41.0
        stages = 8 if case["model"] == "reverso" else 12
        evals = float(n) * case["steps"] * stages
        return dict(bytes=evals * 8 * 12, flops=evals * (per * case["obs"] + 300))
    layers = sum(a * b for a, b in zip(Surrogate().sizes[:-1], Surrogate().sizes[1:]))
    if kind == "predict":
        return dict(bytes=n * (80 + 256 + 8) + 2 * layers, flops=n * (2.0 * layers + 2 * 64 * 64))
    s = case["samples"] // case["batch"] * case["batch"]
    return dict(bytes=s * 74 * 4 + s / case["batch"] * layers * 34, flops=6.0 * s * layers)


# ---------------------------------------------------------------------------
# the same in 64 bits
def _side(X, Y, pa, pb, b):
    """Angular-dislocation pair v(B) - v(A) of one rectangle side for a batch of sources: X, Y are
    (1, M), pa, pb and b (n, 3).  Nikkhoo et al. 2016, surface displacements of the CDM."""
    side = pb - pa
    length, horiz = side.norm(dim=1), side[:, :2].norm(dim=1)
    live = horiz > 1e-12 * length
    c, s = (torch.where(live, side[:, j] / horiz, float(j == 0))[:, None] for j in (0, 1))
    beta0 = torch.atan2(horiz, -side[:, 2])[:, None]
    b1, b2, b3 = c * b[:, :1] + s * b[:, 1:2], s * b[:, :1] - c * b[:, 1:2], -b[:, 2:3]
    y1a = c * (X - pa[:, :1]) + s * (Y - pa[:, 1:2])
    y2 = s * (X - pa[:, :1]) - c * (Y - pa[:, 1:2])
    beta = torch.where(y1a >= 0, beta0 - math.pi, beta0)
    sb, cb = torch.sin(beta), torch.cos(beta)
    cot, coth, k = cb / sb, 1.0 / torch.tan(0.5 * beta), 1.0 - 2.0 * NU

    def one(y1, a):
        z1, z3 = y1 * cb + a * sb, y1 * sb - a * cb
        r = torch.sqrt(y1 * y1 + y2 * y2 + a * a)
        p, q = r + a, r - z3
        F = 2.0 * torch.atan2(y2, p * coth - y1)
        lp, lq = torch.log(p), torch.log(q)
        rq = r * q
        v1 = b1 * ((1 - k * cot ** 2) * F + y2 / p * (k * (cot + y1 / (2 * p)) - y1 / r) - y2 * (r * sb - y1) * cb / rq)
        v1 += b2 * (k * ((cot ** 2 - 0.5) * lp - cot ** 2 * cb * lq)
                    - (k * (y1 * cot + 0.5 * a + y1 * y1 / (2 * p)) - y1 * y1 / r) / p + z1 * (r * sb - y1) / rq)
        v1 += b3 * y2 * (r * sb - y1) * sb / rq
        v2 = b1 * (k * ((0.5 + cot ** 2) * lp - cot / sb * lq)
                   - (k * (y1 * cot - 0.5 * a - y2 * y2 / (2 * p)) + y2 * y2 / r) / p + y2 * y2 * cb / rq)
        v2 += b2 * ((1 + k * cot ** 2) * F - y2 / p * (k * (cot + y1 / (2 * p)) - y1 / r) - y2 * z1 / rq)
        v2 -= b3 * y2 * y2 * sb / rq
        v3 = b1 * (k * F * cot + y2 / p * (2 * NU + a / r) - y2 * cb / q * (cb + a / r))
        v3 += b2 * (-k * cot * (lp - cb * lq) - y1 / p * (2 * NU + a / r) + z1 / q * (cb + a / r))
        v3 += b3 * (F + y2 * (r * cb + a) * sb / rq)
        return v1, v2, v3

    at = one(y1a, -pa[:, 2:3])
    bt = one(y1a - (c * side[:, :1] + s * side[:, 1:2]), -pb[:, 2:3])
    w = torch.where(live, 0.5 / math.pi, 0.0)[:, None]
    v1, v2, v3 = (torch.where(live[:, None], (q - p) * w, 0.0) for p, q in zip(at, bt))
    return c * v1 + s * v2, s * v1 - c * v2, -v3


def _cdm_los(theta, x, y, los):
    """LOS displacements (n, M) of CDM sources in 64 bits."""
    n, m = theta.shape[0], x.numel()
    out = torch.empty(n, m, dtype=torch.float64, device=DEV)
    chunk = max(1, int(1.5e6 // m))
    for i in range(0, n, chunk):
        t = theta[i:i + chunk]
        om = torch.deg2rad(t[:, 7:10])
        (sx, sy, sz), (cx, cy, cz) = (f(om).unbind(1) for f in (torch.sin, torch.cos))
        o, e = torch.zeros_like(cx), torch.ones_like(cx)
        mat = lambda *r: torch.stack(r, 1).view(-1, 3, 3)          # noqa: E731
        R = (mat(cz, sz, o, -sz, cz, o, o, o, e) @ mat(cy, o, -sy, o, e, o, sy, o, cy) @ mat(e, o, o, o, cx, sx, o, -sx, cx))
        ax = R.transpose(1, 2) * t[:, 4:7, None]                    # semi-axis vectors
        centre = torch.stack([t[:, 0], t[:, 1], -t[:, 2]], 1)
        u = [0.0, 0.0, 0.0]
        # the rectangles normal to the body's x, y and z axis, corners in the reference's order
        for f, g in ((ax[:, 1], ax[:, 2]), (-ax[:, 0], ax[:, 2]), (ax[:, 0], ax[:, 1])):
            P = [centre + f + g, centre - f + g, centre - f - g, centre + f - g]
            nrm = torch.linalg.cross(P[1] - P[0], P[3] - P[0])
            b = nrm / nrm.norm(dim=1, keepdim=True) * t[:, 3:4]
            for j in range(4):
                u = [p + q for p, q in zip(u, _side(x[None], y[None], P[j], P[(j + 1) % 4], b))]
        out[i:i + chunk] = u[0] * los[:, 0] + u[1] * los[:, 1] + u[2] * los[:, 2]
    return out


def _mogi_los(theta, x, y, los, sources=1):
    """LOS displacements (n, M) of point sources in 64 bits, log10 ΔV."""
    u = 0.0
    for s in range(sources):
        xs, ys, d, v = theta[:, 4 * s:4 * s + 4, None].unbind(1)
        dx, dy = xs - x, ys - y
        u = u + (NU - 1.0) / math.pi * 10.0 ** v * (dx * los[:, 0] + dy * los[:, 1] - d * los[:, 2]) \
            / (dx * dx + dy * dy + d * d) ** 1.5
    return u


def _misfit(u, inp, off):
    r = u - inp["d"]
    if off.shape[1]:
        r = r - off[:, inp["oid"]]
    m = r.shape[1]
    return -0.5 * m * math.log(2 * math.pi * inp["var"]) - 0.5 * (r * r).sum(1) / inp["var"], r


def _cdm_llk(inp, theta):
    return _misfit(_cdm_los(theta, inp["x"], inp["y"], inp["los"]), inp, theta[:, 10:])


def _reverso_fields(theta, txy):
    """Displacements (n, points, 3) of the two-reservoir model, the default strategy's convention."""
    Q, Hs, Hd, as_, ad, ac = (theta[:, j, None] for j in range(6))
    G, v, mu = REVERSO["G"], REVERSO["v"], REVERSO["mu"]
    k, Hc, gam = (ad / as_) ** 3, Hd - Hs, 8.0 * (1 - v) / (3 * np.pi)
    gr = gam * (1 + k)
    tau = 8 * mu * Hc ** gam * gam * k * as_ ** 3 / (G * ac ** 4 * gr)
    A = gam * k / gr * (REVERSO["drho"] * REVERSO["g"] * Hc - 8 * gam * mu * Q * Hc / (np.pi * ac ** 4 * gr))
    t, x, y = txy.T
    f0, f1 = A * -np.expm1(-t / tau), G * Q * t / (np.pi * as_ ** 3 * gr)
    F, uz = 0.0, 0.0
    for H, a, p in ((Hs, as_, f1 + f0), (Hd, ad, f1 - f0 / k)):
        R2 = x * x + y * y + H * H
        f = 4 * H * H / (np.pi * R2) * a ** 3 * (1 - v) / G / R2 ** 1.5 * p
        F, uz = F + f, uz + H * f
    return np.stack([x * F, y * F, uz], 2)


def _grid_schedule(llk, target=1.0, tol=0.01):
    """δβ from β = 0 by the reference's grid search, its COV and the weights."""
    med, top, n = float(np.median(llk)), float(llk.max()), llk.size

    def cov(g):
        if g * (top - med) > 709.78:
            return 1e100
        w = np.exp(g * (llk - top))
        c = n * math.sqrt(max(0.0, ((w * w).sum() / w.sum() ** 2 - 1 / n) / (n - 1)))
        return c if math.isfinite(c) else 1e100

    low, high, level, found = 0.0, 1.0, 0, False
    if cov(high) < target + tol:
        guess, found = high, True
    while not found and level < 11:
        level += 1
        step = (high - low) / 10.0
        pts = [low]
        for _ in range(10):
            pts.append(pts[-1] + step)
        guess = (pts[-1] + step) - step
        for j, g in enumerate(pts):
            c = cov(g)
            if abs(c - target) < tol or c >= target:
                found, guess = abs(c - target) < tol or j == 0, g
                break
        high, low = guess, guess - step
    w = np.exp(guess * (llk - top))
    return guess, cov(guess), w / w.sum()


def _layers(flat, sizes, half=True):
    """(W, b) of each layer in 64 bits, W as its 16-bit copy holds it."""
    at, out = 0, []
    for fi, fo in zip(sizes[:-1], sizes[1:]):
        W = flat[at:at + fi * fo].view(fo, fi)
        out.append(((W.float().bfloat16() if half else W).double(), flat[at + fi * fo:at + fi * fo + fo].double()))
        at += fi * fo + fo
    return out


def _net(layers, h):
    for i, (W, b) in enumerate(layers):
        h = h @ W.T + b
        if i < len(layers) - 1:
            h = torch.nn.functional.gelu(h)
    return h


def exact(case, seed):
    kind = case["kind"]
    if kind == "cdm":
        if case["chains"] * case["stations"] > 4e7:
            return None
        inp = _cdm_inputs(case, seed)
        theta = inp["theta"]
        llk, r = _cdm_llk(inp, theta)
        if case["call"] == "residuals":
            return {"llk": llk, "residuals": torch.nn.functional.pad(r, (0, -r.shape[1] % 128))}
        if case["call"] == "walk":
            out = ~_below(theta) & (inp["mask"] == 0)
            llk = torch.where(llk < inp["floor"], -math.inf, llk)
            return {"llk": torch.where((inp["mask"] != 0) | out, 0.0, llk), "mask": None}
        return {"llk": llk}
    if kind == "mogi":
        inp = _mogi_inputs(case, seed)
        llk = [_misfit(_mogi_los(t[:, :4], inp["x"], inp["y"], inp["los"]), inp, t[:, 4:])[0]
               for t in inp["theta"].split(1024)]
        return {"llk": torch.cat(llk)}
    if kind == "dense":
        sets, theta = _dense_inputs(case, seed)
        llk = torch.zeros(theta.shape[0], dtype=torch.float64, device=DEV)
        for s in sets:
            L = torch.linalg.cholesky(s["cd"])
            r = _mogi_los(theta, s["x"], s["y"], s["los"], 2) - s["d"]
            z = torch.linalg.solve_triangular(L, r.T, upper=False)
            llk -= 0.5 * (z * z).sum(0) + 0.5 * r.shape[1] * math.log(2 * math.pi) + L.diagonal().log().sum()
        return {"llk": llk}
    if kind == "linear":
        G, d, cd, theta = _linear_inputs(case, seed)
        L = torch.linalg.cholesky(cd)
        A, b = (torch.linalg.solve_triangular(L, v, upper=False) for v in (G, d[:, None]))
        z = theta @ A.T - b.T
        return {"llk": -0.5 * (z * z).sum(1) - 0.5 * d.numel() * math.log(2 * math.pi) - L.diagonal().log().sum()}
    if kind == "cov":
        theta, prior, data = (t.cpu().numpy() for t in _cov_inputs(case, seed))
        none = dict(theta=None, prior=None, data=None, posterior=None)
        if case["solver"] == "brent":
            return dict(beta=None, dbeta_cov=None, w=None, sigma=None, **none)
        db, cov, w = _grid_schedule(data)
        mean = (w[:, None] * theta).sum(0) / w.sum()
        sigma = (theta * w[:, None]).T @ theta - np.outer(mean, mean)
        return dict(beta=np.array([db]), dbeta_cov=np.array([db, cov]), w=w, sigma=sigma, **none)
    if kind == "anneal":
        return None
    sizes, flat = _network(seed)
    if kind == "predict":
        fields, d, theta, lo, hi = _predict_inputs(case, seed)
        # the basis is an input of the prediction: the one the program fitted
        sur = prepare(case, seed)["sur"]
        b = {k: v.double() if torch.is_tensor(v) else v for k, v in sur.basis.items()}
        c = _net(_layers(torch.from_numpy(flat).to(DEV), sizes), 2 * (theta - lo) / (hi - lo) - 1)
        cs = c * b["scale"]
        llk = b["norm"] - 0.5 * (b["q0"] - 2 * cs @ b["h"] + ((cs @ b["G"]) * cs).sum(1))
        return {"llk": llk, "coefficients": c}
    x, y = (t.double() for t in _train_inputs(case, seed))
    flat = torch.from_numpy(flat).to(DEV).double()
    m, v = torch.zeros_like(flat), torch.zeros_like(flat)
    n, B = case["samples"], min(case["batch"], case["samples"])
    order = torch.randperm(n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(0))
    loss = 0.0
    for k, at in enumerate(range(0, n - B + 1, B)):
        sel = order[at:at + B]
        with torch.enable_grad():
            layers = [t.requires_grad_() for pair in _layers(flat, sizes) for t in pair]
            e = _net(list(zip(layers[::2], layers[1::2])), x[sel]) - y[sel]
            part = 0.5 * (e * e).sum() / B
            grads = torch.cat([g.reshape(-1) for g in torch.autograd.grad(part, layers)])
        loss += float(part)
        m, v = 0.9 * m + 0.1 * grads, 0.999 * v + 0.001 * grads * grads
        flat = flat - 1e-3 * (m / (1 - 0.9 ** (k + 1))) / ((v / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"params": flat, "m": m, "v": v, "loss": loss / max(1, n // B)}
