"""Performance cases of the parametric light-curve fitter: the calls a user's
program makes through the public entry points, over the sizes they make them
with.

Whole fits (`Context.fit_batch`) are most of what users run: one alert as it
arrives, a night's hundred, a survey field's thousands, densely sampled
sources, each with the options the API offers (all models, the Bazin-first
gate, the joint multi-band fit, one forced model; SVI or Laplace).  Beside
them stand the separately called stages: the finalisation of fits selected
elsewhere (`Context.finalize_batch`), the swarm-cost and SVI exports that the
reference's GPU host drives (`launch_batch_pso_cost`, `launch_batch_svi_fit`)
and the SVI step's differentiable ELBO (`svi_elbo`).

Sizes are those of the repository's workloads (synth.py, bench.py, tests).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from lightcurve_fitting_gb300 import abi, synth
from lightcurve_fitting_gb300.lib import default_context, load
from lightcurve_fitting_gb300.svi_grad import BandArrays, svi_elbo

# Swarm boxes of the models' internal parameters (the bounds a driver of the
# swarm-cost export draws its particles from).
BOX = [
    ([-3.0, -0.3, -100.0, -2.0, -2.0, -5.0], [3.0, 0.3, 100.0, 5.0, 6.0, 0.0]),
    ([-1.5, -0.02, 1.0, -60.0, -1.0, 1.0, -6.0], [1.5, 0.05, 5.0, 40.0, 3.0, 5.5, 0.0]),
    ([-3.0, -1.0, -100.0, -2.0, -1.0, 0.5, -5.0], [3.0, 1.0, 100.0, 5.0, 6.0, 4.0, 0.0]),
    ([-3.0, -100.0, 0.5, -3.0, -5.0], [3.0, 100.0, 4.5, 3.0, 0.0]),
    ([-3.0, -100.0, 0.0, 0.5, -5.0], [3.0, 100.0, 6.0, 4.5, 0.0]),
    ([-3.0, -100.0, 0.1, -1.0, -5.0], [3.0, 100.0, 3.0, 4.0, 0.0]),
    ([-3.0, -100.0, -2.0, -2.0, 0.5, -5.0], [3.0, 100.0, 6.0, 3.0, 5.0, 0.0]),
]
# A typical fitted parameter vector of each model, t0 (abi.T0_IDX) relative to
# the band's brightest point (MetzgerKN: absolute).
TYPICAL = [
    [0.3, 0.0, -5.0, 1.6, 3.4, -3.0],
    [0.2, 0.005, 2.9, -8.0, 1.4, 3.5, -3.0],
    [0.3, 0.0, -5.0, 1.5, 3.3, 1.67, -3.0],
    [0.6, -15.0, 2.4, 0.0, -3.0],
    [0.6, -15.0, 3.0, 2.3, -3.0],
    [0.4, -4.0, 0.4, 2.6, -3.0],
    [0.3, -6.0, 1.6, 0.5, 2.0, -3.0],
    [-1.75, -1.25, 0.5, -0.5, -2.0],
]


def listed():
    return [
        # One alert of a live stream: latency of a single source's whole fit.
        dict(name="alert", kind="fit", light="uneven", sources=1, points=500, mode="all", method="svi"),
        # The basic workload: 100 sources x 3 x 30, all models, Laplace.
        dict(name="basic_laplace", kind="fit", light="basic", sources=100, points=30, mode="all", method="laplace"),
        # The same sources as `fit_parametric(.., false, Laplace)` fits them: the joint multi-band branch.
        dict(name="basic_joint", kind="fit", light="basic", sources=100, points=30, mode="joint", method="laplace"),
        # A night's batch of an alert broker.
        dict(name="uneven_1k", kind="fit", light="uneven", sources=1000, points=500, mode="all", method="svi"),
        # The headline workload: 10,000 uneven sources, PSO + SVI.
        dict(name="uneven_10k", kind="fit", light="uneven", sources=10000, points=500, mode="all", method="svi"),
        # Densely sampled sources (the precision workload's 2,000 points a band).
        dict(name="long_bands", kind="fit", light="long", sources=96, points=2000, mode="all", method="laplace"),
        # `fit_parametric` with fit_all_models = false on a survey batch: joint fit, then SVI per band.
        dict(name="joint_500", kind="fit", light="uneven", sources=500, points=500, mode="joint", method="svi"),
        # `fit_parametric_model` with the default Bazin-first gate.
        dict(name="gated_1k", kind="fit", light="uneven", sources=1000, points=500, mode="gated", method="svi"),
        # Finalisation of (band, model) pairs selected elsewhere, every model of 600 bands.
        dict(name="finalize", kind="finalize", bands=600, method="svi"),
        # One swarm-cost launch of the reference's GPU host: 30 particles a band, Villar.
        dict(name="swarm_cost", kind="swarm_cost", bands=10000, particles=30, model=1),
        # The reference's GPU SVI call over a batch's selected bands.
        dict(name="svi_export", kind="svi_export", bands=3000, steps=300, samples=4),
        # The gradient workload's ELBO and its gradient: 64 points, 8 samples, 60 observations.
        dict(name="elbo_grad", kind="elbo_grad", points=64, samples=8, model=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit"] * 6 + ["finalize", "swarm_cost", "svi_export", "elbo_grad"])
    if kind == "fit":
        light = rng.choice(["uneven", "uneven", "basic", "long"])
        mode = rng.choice(["all", "all", "joint", "gated", "forced"])
        method = rng.choice(["svi", "laplace"])
        if light == "long":
            points = _log_int(rng, 300, 2000)
            sources = _log_int(rng, 1, max(2, 60 * 2000 // points))
        elif light == "basic":
            points = _log_int(rng, 10, 100)
            sources = _log_int(rng, 1, 2000)
        else:
            points = rng.choice([100, 500, 1000])
            sources = _log_int(rng, 1, 1500 if mode == "joint" else 6000)
        if mode == "joint":
            sources = min(sources, 1500)
            if light == "long":
                sources = min(sources, 40)
        case = dict(kind=kind, light=light, sources=sources, points=points, mode=mode, method=method)
        if mode == "forced":
            case["model"] = rng.randrange(8)
        return case
    if kind == "finalize":
        return dict(kind=kind, bands=_log_int(rng, 1, 3000), method=rng.choice(["svi", "laplace"]))
    if kind == "swarm_cost":
        return dict(kind=kind, bands=_log_int(rng, 3, 20000), particles=rng.choice([1, 7, 30, 40]), model=rng.randrange(7))
    if kind == "svi_export":
        return dict(kind=kind, bands=_log_int(rng, 1, 4000), steps=rng.choice([50, 200, 500]), samples=rng.choice([1, 4, 8]))
    return dict(kind=kind, points=_log_int(rng, 1, 4000), samples=rng.choice([1, 4, 8]), model=rng.randrange(7))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _photometry(case, seed):
    n, points = case["sources"], case["points"]
    if case["light"] == "uneven":
        return synth.config_uneven(n, seed=seed, max_count=points)
    if case["light"] == "basic":
        return synth.generate(n, np.full((n, 3), points), np.zeros(n, np.int64), seed=seed, t_span=150.0,
                              drop_nights=0.0, name="basic")
    return synth.generate(n, np.full((n, 3), points), np.zeros(n, np.int64), seed=seed, t_span=1000.0,
                          drop_nights=0.0, amp_lo=10.0, amp_hi=1.0e6, name="long")


def _typical(rng, model, t_peak, scatter):
    p = np.array(TYPICAL[model])
    if model != 7:
        p[abi.T0_IDX[model]] += t_peak
    return p + scatter * rng.standard_normal(p.size)


def _pairs(n_bands, seed):
    """(band, model) pairs of every model over `n_bands` bands of an uneven
    batch: a CSR batch whose sources are the pairs, the models and parameters."""
    base = synth.config_uneven(-(-n_bands // 3) + 4, seed=seed)
    rng = np.random.default_rng(seed + 17)
    bands = [b for s in range(base.n_sources) for b in base.bands_of(s) if b[0].size >= 5][:n_bands]
    t, f, e, bo, model, params = [], [], [], [0], [], []
    for bt, bf, be in bands:
        peak = bt[np.argmax(bf)]
        for m in range(8):
            t.append(bt)
            f.append(bf)
            e.append(be)
            bo.append(bo[-1] + bt.size)
            model.append(m)
            row = np.full(7, np.nan)
            p = _typical(rng, m, peak, 0.05)
            row[:p.size] = p
            params.append(row)
    n = len(model)
    batch = synth.PhotometryBatch(np.concatenate(t), np.concatenate(f), np.concatenate(e), np.asarray(bo, np.int64),
                                  np.arange(n + 1, dtype=np.int32), np.zeros(n, np.int32), "pairs")
    return batch, np.asarray(model, np.int32), np.asarray(params)


def _gpu_sources(n_bands, seed):
    """Bands of an uneven batch as the exports take them: peak-normalised
    device arrays, int32 offsets and the host copies."""
    base = synth.config_uneven(-(-n_bands // 3) + 4, seed=seed)
    cnt = base.band_counts()
    keep = np.flatnonzero(cnt > 0)[:n_bands]
    idx = np.concatenate([np.arange(base.band_obs_offsets[b], base.band_obs_offsets[b + 1]) for b in keep])
    n = cnt[keep]
    offs = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
    t, f, e = base.times[idx], base.flux[idx], base.flux_err[idx]
    peak = np.repeat(np.maximum.reduceat(f, offs[:-1]), n)
    t_peak = np.array([t[a + np.argmax(f[a:b])] for a, b in zip(offs[:-1], offs[1:])])
    host = dict(t=t, f=f / peak, var=(e / peak) ** 2 + 1e-10, up=(f / e < 3.0).astype(np.int32), uf=3.0 * e / peak,
                offs=offs)
    return host, t_peak


def _cost_inputs(case, seed):
    host, t_peak = _gpu_sources(case["bands"], seed)
    nb, m = host["offs"].size - 1, case["model"]
    rng = np.random.default_rng(seed + 29)
    lo, hi = np.array(BOX[m][0]), np.array(BOX[m][1])
    pos = rng.uniform(lo, hi, (nb, case["particles"], lo.size))
    # a swarm under way: t0 near the band's light curve, amplitudes near one
    i0 = abi.T0_IDX[m]
    pos[:, :, i0] = np.clip(t_peak[:, None] + rng.uniform(-30.0, 10.0, pos.shape[:2]), lo[i0], hi[i0])
    pos[:, :, 0] = rng.uniform(-1.0, 1.0, pos.shape[:2])
    return host, pos


def _svi_inputs(case, seed):
    host, t_peak = _gpu_sources(case["bands"], seed)
    nb = host["offs"].size - 1
    rng = np.random.default_rng(seed + 31)
    models = rng.integers(0, 7, nb).astype(np.int32)
    init, width = np.zeros((nb, 7)), np.ones((nb, 7))
    for i, m in enumerate(models):
        p = _typical(rng, m, t_peak[i], 0.05)
        init[i, :p.size] = p
        width[i, :p.size] = 2.0
    nps = np.array([abi.N_PARAMS[m] for m in models], np.int32)
    ses = np.array([abi.SE_IDX[m] for m in models], np.int32)
    return host, models, nps, ses, init, width


def _elbo_inputs(case, seed):
    base = synth.config_gradient(8, seed=seed)
    band = BandArrays(*next(b for s in range(base.n_sources) for b in base.bands_of(s) if b[0].size >= 50))
    rng = np.random.default_rng(seed + 37)
    m, n = case["model"], case["points"]
    npar = abi.N_PARAMS[m]
    init = _typical(rng, m, band.times[np.argmax(band.flux)], 0.0)
    init[abi.SE_IDX[m]] = -2.0  # early in an SVI run: the fit's extra scatter is still wide
    mu = init + 0.1 * rng.standard_normal((n, npar))
    var = np.concatenate([mu, rng.uniform(-4.0, -1.5, (n, npar))], axis=1)
    eps = rng.standard_normal((n, case["samples"], npar))
    return band, init, var, eps


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fit":
        return dict(case=case, ctx=default_context(), batch=_photometry(case, seed))
    if kind == "finalize":
        batch, model, params = _pairs(case["bands"], seed)
        return dict(case=case, ctx=default_context(), batch=batch, model=model, params=params)
    if kind == "elbo_grad":
        band, init, var, eps = _elbo_inputs(case, seed)
        v = torch.tensor(var, device="cuda", requires_grad=True)
        return dict(case=case, ctx=default_context(), band=band, init=init, var=v, eps=eps)
    dev = lambda a: torch.tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    if kind == "swarm_cost":
        host, pos = _cost_inputs(case, seed)
        out = torch.empty(pos.shape[:2], dtype=torch.float64, device="cuda")
        return dict(case=case, lib=load(), obs=[dev(host[k]) for k in ("t", "f", "var", "up", "uf", "offs")],
                    pos=dev(pos), out=out)
    host, models, nps, ses, init, width = _svi_inputs(case, seed)
    outs = [torch.empty(init.shape, dtype=torch.float64, device="cuda") for _ in range(2)]
    outs.append(torch.empty(init.shape[0], dtype=torch.float64, device="cuda"))
    return dict(case=case, lib=load(), obs=[dev(host[k]) for k in ("t", "f", "var", "up", "uf", "offs")],
                args=[dev(a) for a in (init, models, nps, ses, init, width)], outs=outs)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _arrays(res):
    return {name: getattr(res, name) for name, _ in abi.FitOutputs._fields_}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fit":
        mode = case["mode"]
        res = state["ctx"].fit_batch(
            state["batch"], fit_all_models=mode == "all",
            method=abi.METHOD_SVI if case["method"] == "svi" else abi.METHOD_LAPLACE,
            forced_model=case["model"] if mode == "forced" else -1, joint_multiband=mode == "joint")
        return _arrays(res)
    if kind == "finalize":
        res = state["ctx"].finalize_batch(
            state["batch"], state["model"], state["params"],
            method=abi.METHOD_SVI if case["method"] == "svi" else abi.METHOD_LAPLACE)
        return _arrays(res)
    if kind == "elbo_grad":
        var = state["var"]
        elbo, flags = svi_elbo(var, state["band"], case["model"], state["init"], state["eps"], state["ctx"])
        (grad,) = torch.autograd.grad(elbo.sum(), var)
        return dict(elbo=elbo.detach(), grad=grad, flags=flags)
    obs = [x.data_ptr() for x in state["obs"]]
    if kind == "swarm_cost":
        pos, out = state["pos"], state["out"]
        n, k, d = pos.shape
        state["lib"].launch_batch_pso_cost(*obs, pos.data_ptr(), out.data_ptr(), n, k, d, case["model"], 1, 256)
        return dict(costs=out)
    args, outs = state["args"], state["outs"]
    n, d = args[0].shape
    state["lib"].launch_batch_svi_fit(*obs, *[x.data_ptr() for x in args], *[x.data_ptr() for x in outs], n, d,
                                      case["steps"], case["samples"], 0.01, 1, 256)
    return dict(mu=outs[0], log_sigma=outs[1], elbo=outs[2])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
EVAL = 30.0       # operations of one model evaluation and its likelihood term
EVAL_GRAD = 80.0  # the same with the gradient
MEAN_UNEVEN = 55.0


def work(case):
    kind = case["kind"]
    if kind == "fit":
        n_src = case["sources"]
        obs = 3.0 * n_src * (min(MEAN_UNEVEN, case["points"]) if case["light"] == "uneven" else 0.8 * case["points"])
        mode = case["mode"]
        iters = 40.0  # of the swarm's 60, before it stalls
        swarm = 30.0 * iters * EVAL
        models = {"all": 8.0, "gated": 3.0, "forced": 1.0, "joint": 0.0}[mode]
        flops = obs * models * (3.0 * swarm + 150.0 * EVAL_GRAD)
        if mode == "joint":
            flops += obs * 3.0 * 200.0 * 400.0 * EVAL
        flops += obs / 3.0 * 2.0 * swarm * (1.0 + 2.0 + 3.0 + 4.0)  # MultiBazin of the longest band
        if case["method"] == "svi":
            flops += obs * 600.0 * 4.0 * EVAL_GRAD + obs / 3.0 * 8.0 * swarm  # SVI, profile t0 search
        else:
            flops += obs * 6.0 * 2.0 * EVAL_GRAD
        flops += obs * 140.0 * EVAL
        per_band = 8.0 * (7 * 3 + 4 + 8 + 18 + 10) + 16.0 + (8.0 * 56 if mode == "all" else 0.0)
        return {"bytes": obs * 24.0 + 3.0 * n_src * (per_band + 8.0), "flops": flops}
    if kind == "finalize":
        obs = case["bands"] * 8.0 * MEAN_UNEVEN
        fit = 600.0 * 4.0 * EVAL_GRAD if case["method"] == "svi" else 6.0 * 2.0 * EVAL_GRAD
        return {"bytes": obs * 24.0 + case["bands"] * 8.0 * 8.0 * 60.0, "flops": obs * (fit + 140.0 * EVAL)}
    if kind == "elbo_grad":
        d = abi.N_PARAMS[case["model"]]
        return {"bytes": 50.0 * 36.0 + case["points"] * 8.0 * (4 * d + 1 + case["samples"] * d),
                "flops": case["points"] * case["samples"] * 50.0 * EVAL_GRAD}
    obs = case["bands"] * MEAN_UNEVEN
    if kind == "swarm_cost":
        rows = case["bands"] * case["particles"]
        return {"bytes": obs * 36.0 + rows * 8.0 * (abi.N_PARAMS[case["model"]] + 1.0),
                "flops": obs * case["particles"] * EVAL}
    return {"bytes": obs * 36.0 + case["bands"] * 8.0 * 36.0, "flops": obs * 0.7 * case["steps"] * case["samples"] * EVAL_GRAD}


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch on the host
# ---------------------------------------------------------------------------
def _flux(m, p, t):
    """Model m at times t; p: parameters along the last axis."""
    g = lambda k: p[..., k]  # noqa: E731
    sigmoid = lambda x: 1.0 / (1.0 + torch.exp(-x))  # noqa: E731
    soft = lambda x: torch.log(1.0 + torch.exp(x)) + 1e-6  # noqa: E731
    a = torch.exp(g(0))
    if m == 0:
        dt = t - g(2)
        return a * torch.exp(-dt / torch.exp(g(4))) * sigmoid(dt / torch.exp(g(3))) + g(1)
    if m == 1:
        beta, gamma, ph, tf = g(1), torch.exp(g(2)), t - g(3), torch.exp(g(5))
        w = sigmoid(10.0 * (ph - gamma))
        late = (1.0 - beta * gamma) * torch.exp((gamma - ph) / tf)
        return a * sigmoid(ph / torch.exp(g(4))) * ((1.0 - w) * (1.0 - beta * ph) + w * late)
    if m == 2:
        ph = t - g(2)
        return a * sigmoid(ph / torch.exp(g(3))) * torch.pow(1.0 + soft(ph) / torch.exp(g(4)), -g(5)) + g(1)
    ps = soft(t - g(1))
    if m == 3:
        f, x = sigmoid(g(3)), ps / torch.exp(g(2))
        return a * (f * torch.exp(-ps / 8.8) + (1.0 - f) * torch.exp(-ps / 111.3)) * (1.0 - torch.exp(-x * x))
    if m == 4:
        w, x = 1.0 + ps / torch.exp(g(2)), ps / torch.exp(g(3))
        return a / (w * w) * (1.0 - torch.exp(-x * x))
    if m == 5:
        r = ps / torch.exp(g(3))
        return a * sigmoid(5.0 * (t - g(1))) * torch.pow(ps, -g(2)) * torch.exp(-r * r)
    lr = torch.log(ps / torch.exp(g(2)))
    return a * torch.pow(torch.exp(2.0 * g(3) * lr) + torch.exp(2.0 * g(4) * lr), -0.5)


def _log_cdf(x):
    """ln Phi(x) by Abramowitz & Stegun 7.1.26, the fitter's definition."""
    z = -x * math.sqrt(0.5)
    t = 1.0 / (1.0 + 0.3275911 * z.abs())
    poly = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))))
    e = poly * torch.exp(-z * z)
    phi = torch.where(z >= 0, 0.5 * e, 1.0 - 0.5 * e).clamp_min(1e-300)
    far = torch.where(x < -30.0, -x, torch.ones_like(x))
    tail = -0.5 * x * x - 0.5 * math.log(2.0 * math.pi) - torch.log(far)
    return torch.where(x > 8.0, torch.zeros_like(x), torch.where(x < -30.0, tail, torch.log(phi)))


def _exact_cost(case, seed):
    host, pos = _cost_inputs(case, seed)
    n = np.diff(host["offs"])
    rows = torch.tensor(pos)
    total = torch.zeros(rows.shape[:2], dtype=torch.float64)
    bad = torch.zeros(rows.shape[:2], dtype=torch.bool)
    c = {k: torch.tensor(v) for k, v in host.items()}
    for i in range(int(n.max())):  # the i-th observation of every band that has one
        b = torch.tensor(np.flatnonzero(n > i))
        o = c["offs"][b].long() + i
        col = lambda k: c[k][o][:, None]  # noqa: E731
        p = rows[b]
        pred = _flux(case["model"], p, col("t"))
        tv = col("var") + torch.exp(p[..., -1]) ** 2
        d = pred - col("f")
        term = torch.where(col("up") != 0, -_log_cdf((col("uf") - pred) / torch.sqrt(tv)), d * d / tv + torch.log(tv))
        bad[b] |= ~torch.isfinite(pred)
        total[b] += torch.where(torch.isfinite(pred), term, torch.zeros_like(term))
    cost = total / torch.tensor(n)[:, None]
    return dict(costs=torch.where(bad, torch.full_like(cost, 1e99), cost))


# Widths of the SVI's Gaussian prior by model, centred on the initial
# parameters; sigma_extra is centred on PRIOR_SE.
PRIOR_WIDTH = [
    [2, 2, 2, 2, 2, 2], [2, 2, 2, 2, 2, 2, 2], [2, 2, 2, 2, 2, 1, 2], [2, 2, 1, 2, 2], [2, 2, 1.5, 1, 2],
    [2, 2, 1, 2, 2], [2, 2, 2, 1, 1, 2],
]
PRIOR_SE = 0.0


def _exact_elbo(case, seed):
    band, init, var, eps = _elbo_inputs(case, seed)
    m, np_ = case["model"], abi.N_PARAMS[case["model"]]
    vp = torch.tensor(var, requires_grad=True)
    mu, ls, e = vp[:, :np_], vp[:, np_:], torch.tensor(eps)
    theta = mu[:, None, :] + torch.exp(ls)[:, None, :] * e  # [points, samples, np]
    t, f, v, uf = (torch.tensor(x) for x in (band.times, band.flux, band.obs_var, band.upper_flux))
    up = torch.tensor(band.is_upper) != 0
    th = theta[:, :, None, :]
    pred = _flux(m, th, t)
    tv = v + torch.exp(2.0 * th[..., abi.SE_IDX[m]])
    det = -0.5 * ((f - pred) ** 2 / tv + torch.log(2.0 * math.pi * tv))
    # an upper limit's gradient is the Gaussian density over the A&S CDF in
    # its 1 + erf form, not the derivative of the A&S expression
    z = (uf - pred) / torch.sqrt(tv)
    with torch.no_grad():
        w = z * math.sqrt(0.5)
        k = 1.0 / (1.0 + 0.3275911 * w.abs())
        poly = k * (0.254829592 + k * (-0.284496736 + k * (1.421413741 + k * (-1.453152027 + k * 1.061405429))))
        erf = torch.sign(w) * (1.0 - poly * torch.exp(-w * w))
        cdf = (0.5 * (1.0 + erf)).clamp_min(1e-300)
        ratio = torch.exp(-0.5 * z * z) / math.sqrt(2.0 * math.pi) / cdf
    lim = _log_cdf(z.detach()) + ratio * (z - z.detach())
    ok = torch.isfinite(pred)
    ll = torch.where(ok, torch.where(up, lim, det), torch.zeros_like(det)).sum(-1)
    centre = torch.tensor(np.array(init))
    centre[abi.SE_IDX[m]] = PRIOR_SE
    width = torch.tensor(PRIOR_WIDTH[m], dtype=torch.float64)
    lp = (-0.5 * ((theta - centre) / width) ** 2).sum(-1)
    entropy = ls.sum(-1) + 0.5 * np_ * math.log(2.0 * math.pi * 2.71828182845904523536)
    elbo = (ll + lp).mean(-1) + entropy
    (grad,) = torch.autograd.grad(elbo.sum(), vp)
    return dict(elbo=elbo.detach(), grad=grad, flags=None)


def exact(case, seed):
    if case["kind"] == "swarm_cost":
        return _exact_cost(case, seed)
    if case["kind"] == "elbo_grad":
        return _exact_elbo(case, seed)
    # The fits, the finalisation and the SVI export end hundreds of swarm and
    # Adam steps that amplify the last bit: no 64-bit value of their own.
    return None
