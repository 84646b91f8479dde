"""The work that is timed: what a user of the package has it do, from a four-chain call to thousands of chains.

A case is one pass through the public entry points.  Three kinds of call stand for a user's program:

  sample     kernel.sample(state): one transition per call, from the state a program holds
  run        MCMC.run from a post-warmup state, draws kept on the device
  warmup     MCMC.warmup from scratch: init_to_uniform, step size and mass matrix adaptation
  potential  kernel.potential_and_grad(z): the potential and its gradient at given points

over the four model families.  The data, the points and the adapted quantities (step size, inverse mass
matrix) are made from the seed, near the posterior, with the scales that warmup finds.
"""
import math

import numpy as np
import torch

from numpyro_gb300 import HMC, MCMC, NUTS, datasets, models

LOG_2PI = math.log(2.0 * math.pi)


def listed():
    return [
        # the smallest call: numpyro's eight schools with four chains, a program that steps the kernel itself
        {"name": "schools_sample", "family": "hier", "call": "sample", "models": 1, "jmin": 8, "jmax": 8, "per": 4,
         "steps": 10},
        # eight schools as most users run it: four chains, draws after warmup
        {"name": "schools_run", "family": "hier", "call": "run", "models": 1, "jmin": 8, "jmax": 8, "per": 4,
         "samples": 200, "steps": 12},
        # warmup with a dense mass matrix, 64 chains of a 30-group model
        {"name": "hier_warmup_dense", "family": "hier", "call": "warmup", "models": 1, "jmin": 30, "jmax": 30,
         "per": 64, "warmup": 100, "dense": True, "steps": 40},
        # the batch of 4,096 uneven datasets, four chains each, in one persistent launch
        {"name": "uneven_run", "family": "hier", "call": "run", "models": 4096, "jmin": 4, "jmax": 256, "per": 4,
         "samples": 5, "steps": 10},
        # covtype-shaped logistic regression, 1,024 chains on the tensor cores: the headline benchmark
        {"name": "logreg_tc_run", "family": "logreg", "call": "run", "n": 581012, "p": 55, "chains": 1024,
         "precision": "bf16x3", "samples": 2, "steps": 15},
        # the same potential in the default precision
        {"name": "logreg_fp32_potential", "family": "logreg", "call": "potential", "n": 581012, "p": 55,
         "chains": 1024, "precision": "fp32"},
        # a small data set with four chains in the default precision: one launch pair per leapfrog step
        {"name": "logreg_fp32_run", "family": "logreg", "call": "run", "n": 20011, "p": 13, "chains": 4,
         "precision": "fp32", "samples": 10, "steps": 7},
        # horseshoe regression, 256 chains, non-centred, tensor cores: fixed-length HMC
        {"name": "horseshoe_tc_run", "family": "horseshoe", "call": "run", "n": 2000, "p": 1000, "chains": 256,
         "precision": "bf16x3", "noncentered": True, "samples": 3, "steps": 32},
        # the horseshoe potential in the default precision, centred
        {"name": "horseshoe_fp32_potential", "family": "horseshoe", "call": "potential", "n": 2000, "p": 1000,
         "chains": 256, "precision": "fp32", "noncentered": False},
        # stochastic volatility, the benchmark's 256 chains of 4,098 dimensions
        {"name": "sv_run", "family": "sv", "call": "run", "t": 4096, "chains": 256, "noncentered": False,
         "samples": 1, "steps": 900},
        # the non-centred walk with few chains and an odd length
        {"name": "sv_nc_run", "family": "sv", "call": "run", "t": 1001, "chains": 16, "noncentered": True,
         "samples": 2, "steps": 150},
        # the walk's gradient at many points
        {"name": "sv_nc_potential", "family": "sv", "call": "potential", "t": 4096, "chains": 1024,
         "noncentered": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["hier", "hier", "logreg", "logreg", "horseshoe", "sv"])
    if family == "hier":
        call = rng.choice(["sample", "run", "warmup"])
        if call == "run":
            jmax = rng.randint(5, 256)
            return {"family": family, "call": call, "models": _log_int(rng, 1, 4096), "jmin": rng.randint(4, jmax),
                    "jmax": jmax, "per": 4, "samples": rng.randint(2, 5), "steps": 10}
        j = _log_int(rng, 4, 100)
        case = {"family": family, "call": call, "models": 1, "jmin": j, "jmax": j, "per": _log_int(rng, 1, 100),
                "steps": 9}
        if call == "warmup":
            case.update(warmup=rng.randint(40, 120), dense=rng.random() < 0.5 and j <= 40)
        return case
    if family == "logreg":
        case = {"family": family, "call": rng.choice(["run", "potential"]), "p": rng.randint(3, 64),
                "precision": rng.choice(["fp32", "bf16x3"])}
        top = 500000 if case["call"] == "potential" else 100000
        case["n"] = _log_int(rng, 200, top)
        case["chains"] = _log_int(rng, 1, 1024 if case["call"] == "potential" or case["precision"] == "bf16x3" else 128)
        if case["call"] == "run":
            case.update(samples=2, steps=9)
        return case
    if family == "horseshoe":
        case = {"family": family, "call": rng.choice(["run", "potential"]), "n": _log_int(rng, 50, 2000),
                "p": _log_int(rng, 20, 1000), "chains": _log_int(rng, 1, 256),
                "precision": rng.choice(["fp32", "bf16x3"]), "noncentered": rng.random() < 0.5}
        if case["call"] == "run":
            case.update(samples=2, steps=rng.randint(5, 32), noncentered=True)
        return case
    case = {"family": family, "call": rng.choice(["run", "potential"]), "t": _log_int(rng, 100, 4096),
            "chains": _log_int(rng, 1, 256), "noncentered": rng.random() < 0.5}
    if case["call"] == "run":
        case.update(samples=1, steps=255)
        if case["noncentered"]:  # the longest trees
            case.update(t=_log_int(rng, 100, 1500), chains=_log_int(rng, 1, 64))
    return case


# ------------------------------------------------------------------ data and points


def _hier_points(sets, per, dim, g):
    """Near each dataset's posterior: positions, and the variances of one coordinate given the others
    as the inverse mass matrix, [chains, dim]."""
    z = np.zeros((len(sets) * per, dim), np.float32)
    inv = np.ones_like(z)
    for k, (y, s) in enumerate(sets):
        y, v = y.astype(np.float64), s.astype(np.float64) ** 2
        J = y.size
        w = 1.0 / (v + 9.0)
        mu = float((w * y).sum() / w.sum()) * 0.9
        tau2 = max(float(np.mean((y - mu) ** 2 - v)), 1.0)
        tau = math.sqrt(tau2)
        shrink = 1.0 / (1.0 + tau2 / v)
        base = (y - mu) / tau * (1.0 - shrink)
        rows = slice(k * per, (k + 1) * per)
        var_mu = 1.0 / (0.04 + (1.0 / v).sum())
        var_lt = 1.0 / (1.0 + (tau2 * (base ** 2 + shrink) / v).sum())
        z[rows, 0] = mu + math.sqrt(var_mu) * g.standard_normal(per)
        z[rows, 1] = math.log(tau) + math.sqrt(var_lt) * g.standard_normal(per)
        z[rows, 2:2 + J] = base + np.sqrt(shrink) * g.standard_normal((per, J))
        inv[rows, 0], inv[rows, 1], inv[rows, 2:2 + J] = var_mu, var_lt, shrink
    return z, inv


def _logreg_data(case, seed):
    """Continuous, binary and intercept columns as in datasets.covtype_like, made on the GPU."""
    n, p = case["n"], case["p"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    cont = max(1, p // 5)
    X = torch.empty(n, p, device="cuda")
    X[:, :cont] = torch.randn(n, cont, device="cuda", generator=g).bfloat16().float()
    X[:, cont:p - 1] = (torch.rand(n, p - 1 - cont, device="cuda", generator=g) < 0.05).float()
    X[:, p - 1] = 1.0
    beta = torch.randn(p, device="cuda", generator=g) / math.sqrt(p)
    y = (torch.rand(n, device="cuda", generator=g) < torch.sigmoid(X @ beta)).float()
    info = 0.2 * n * torch.tensor([1.0] * cont + [0.05] * (p - 1 - cont) + [1.0], device="cuda") + 1.0
    sd = info.rsqrt()
    z = beta + sd * torch.randn(case["chains"], p, device="cuda", generator=g)
    return X, y, z, (sd ** 2).cpu().numpy()


def _horseshoe_data(case, seed):
    n, p, chains = case["n"], case["p"], case["chains"]
    X, y, beta = datasets.horseshoe_data(seed=seed, n=n, p=p, nonzero=min(10, p // 2))
    g = np.random.default_rng(seed + 1)
    big = beta != 0.0
    tau = 0.01
    lam = np.where(big, 0.0, 0.5) * g.standard_normal((chains, p)) + np.where(big, np.log(np.abs(beta) / tau + 1e-30), 0.0)
    lsig, ltau = 0.02 * g.standard_normal((chains, 1)), math.log(tau) + 0.1 * g.standard_normal((chains, 1))
    eta = np.where(big, np.sign(beta) * np.exp(-(ltau - math.log(tau))), g.standard_normal((chains, p)))
    if case["noncentered"]:
        z = np.concatenate([lam, lsig, ltau, eta], axis=1)
    else:
        z = np.concatenate([np.exp(ltau + lam) * eta, lam, lsig, ltau], axis=1)
    return X, y, z.astype(np.float32)


def _sv_scale(T):
    s0, ramp = 0.03, 1
    for _ in range(8):
        ramp = min(T, max(1, round(2.14 / s0)))
        s0 = math.sqrt(4e-4 + 21.0 / (ramp * T))
    return s0, ramp


def _sv_data(case, seed):
    T, chains = case["t"], case["chains"]
    r, h = datasets.sv_returns(seed=seed, T=T)
    g = np.random.default_rng(seed + 1)
    # the walk starts at 0 and the data at log 0.01: the posterior climbs down over about ramp steps
    s0, ramp = _sv_scale(T)
    h = h * np.minimum(1.0, np.arange(1, T + 1) / ramp)
    z = np.empty((chains, T + 2))
    z[:, T] = math.log(8.0) + 0.2 * g.standard_normal(chains)
    z[:, T + 1] = math.log(s0) + g.standard_normal(chains) / math.sqrt(2.0 * T)
    inv = np.empty(T + 2, np.float32)
    inv[T], inv[T + 1] = 0.1, 0.5 / T
    if case["noncentered"]:
        steps = np.diff(h, prepend=0.0)
        z[:, :T] = steps / np.exp(z[:, T + 1:T + 2]) + 0.1 * g.standard_normal((chains, T))
        inv[:T] = 1.0
    else:
        z[:, :T] = h + 0.2 * s0 * g.standard_normal((chains, T))
        inv[:T] = 0.5 * s0
    return r, z.astype(np.float32), inv


def _step_size(case):
    if case["family"] == "hier":
        return 0.4
    if case["family"] == "logreg":
        return 0.4
    if case["family"] == "horseshoe":
        return 0.002
    # the non-centred walk's stiffest direction moves all T steps together
    return min(0.25, 0.65 / (_sv_scale(case["t"])[0] * case["t"])) if case["noncentered"] else 0.025


def _hier_sets(case, seed):
    jmin, jmax = case["jmin"], case["jmax"]
    sets = datasets.uneven_hierarchical(seed=seed, num_models=1, jmin=jmax, jmax=jmax)  # one of the largest size
    return sets + datasets.uneven_hierarchical(seed=seed + 1, num_models=case["models"] - 1, jmin=jmin, jmax=jmax)


def _data(case, seed):
    """(model, starting points, inverse mass matrix)"""
    if case["family"] == "hier":
        sets = _hier_sets(case, seed)
        model = models.HierarchicalNormal(datasets=sets)
        return (model,) + _hier_points(sets, case["per"], model.latent_dim, np.random.default_rng(seed + 1))
    if case["family"] == "logreg":
        X, y, z, inv = _logreg_data(case, seed)
        return models.LogisticRegression(X.cpu().numpy(), y.cpu().numpy()), z.cpu().numpy(), inv
    if case["family"] == "horseshoe":
        X, y, z = _horseshoe_data(case, seed)
        return models.HorseshoeRegression(X, y, noncentered=case["noncentered"]), z, None
    r, z, inv = _sv_data(case, seed)
    return models.StochasticVolatility(r, noncentered=case["noncentered"]), z, inv


def prepare(case, seed):
    model, z, inv = _data(case, seed)
    chains, call = z.shape[0], case["call"]
    more = {"precision": case.get("precision", "fp32"), "num_chains": chains}
    if call == "warmup":
        kernel = NUTS(model, dense_mass=case["dense"], **more)
        mcmc = MCMC(kernel, num_warmup=case["warmup"], num_samples=1, num_chains=chains, keep_on_device=True)
        return {"call": call, "mcmc": mcmc, "seed": seed}
    if call == "potential":
        kernel = NUTS(model, **more)
        kernel.init(seed, 0, z)
        return {"call": call, "kernel": kernel, "z": torch.as_tensor(z, device="cuda")}
    more.update(step_size=_step_size(case), inverse_mass_matrix=inv, adapt_step_size=False, adapt_mass_matrix=False)
    if case["family"] == "horseshoe":
        kernel = HMC(model, num_steps=case["steps"], trajectory_length=None, **more)
    else:
        kernel = NUTS(model, **more)
    state = kernel.init(seed, 0, z)
    if call == "sample":
        return {"call": call, "kernel": kernel, "state": state}
    mcmc = MCMC(kernel, num_warmup=0, num_samples=case["samples"], num_chains=chains, keep_on_device=True)
    mcmc.post_warmup_state = state
    return {"call": call, "mcmc": mcmc, "seed": seed}


def _state_out(state):
    a = state.adapt_state
    return {"i": state.i, "z": state.z, "z_grad": state.z_grad, "potential_energy": state.potential_energy,
            "energy": state.energy, "num_steps": state.num_steps, "accept_prob": state.accept_prob,
            "mean_accept_prob": state.mean_accept_prob, "diverging": state.diverging, "step_size": a.step_size,
            "inverse_mass_matrix": a.inverse_mass_matrix}


def run(state):
    if state["call"] == "potential":
        return state["kernel"].potential_and_grad(state["z"])
    if state["call"] == "sample":
        return _state_out(state["kernel"].sample(state["state"]))
    mcmc = state["mcmc"]
    if state["call"] == "warmup":
        mcmc.warmup(state["seed"])
        return _state_out(mcmc.last_state)
    mcmc.run(state["seed"], extra_fields=("num_steps", "accept_prob"))
    return {"samples": mcmc.get_samples(group_by_chain=True), "fields": mcmc.get_extra_fields(group_by_chain=True),
            "state": _state_out(mcmc.last_state)}


# ------------------------------------------------------------------ work and reference values


def _sizes(case):
    """(chains, mean latent dimension, data bytes, flops of one potential and gradient over all chains)"""
    if case["family"] == "hier":
        j = 0.5 * (case["jmin"] + case["jmax"])
        chains = case["models"] * case["per"]
        return chains, j + 2.0, 8.0 * j * case["models"], 16.0 * j * chains
    if case["family"] == "sv":
        return case["chains"], case["t"] + 2.0, 4.0 * case["t"], 30.0 * case["t"] * case["chains"]
    n, p, chains = case["n"], case["p"], case["chains"]
    dim = p if case["family"] == "logreg" else 2 * p + 2
    half = case["family"] == "logreg" and case["precision"] == "bf16x3"  # the design matrix is exact in bfloat16
    return chains, float(dim), (2.0 if half else 4.0) * n * p + 4.0 * n, 4.0 * n * p * chains


def work(case):
    chains, dim, data, flops = _sizes(case)
    if case["call"] == "potential":
        return {"bytes": data + chains * (8.0 * dim + 8.0), "flops": flops}
    iterations = {"sample": 1, "run": case.get("samples", 1), "warmup": case.get("warmup", 1)}[case["call"]]
    leaves = iterations * case["steps"]  # leapfrog steps a chain takes, about (exactly for fixed-length HMC)
    mass = dim * dim if case.get("dense") else dim
    state = chains * (16.0 * dim + 8.0 * mass + 60.0)  # position, gradient and mass matrix, read and written
    draws = chains * iterations * (4.0 * dim + 9.0) if case["call"] == "run" else 0.0
    return {"bytes": data + state + draws, "flops": leaves * (flops + chains * (14.0 * dim + 2.0 * mass))}


def _exact_logreg(X, y, z):
    X, y, z = X.double(), y.double(), z.double()
    l = z @ X.T
    pe = (torch.nn.functional.softplus(l) - l * y).sum(1) + 0.5 * (z ** 2).sum(1) + 0.5 * z.shape[1] * LOG_2PI
    return pe, (torch.sigmoid(l) - y) @ X + z


def _exact_horseshoe(case, X, y, z):
    X, y, z = (torch.as_tensor(v, device="cuda").double() for v in (X, y, z))
    n, p = X.shape
    if case["noncentered"]:
        ll, ls, lt, eta = z[:, :p], z[:, p], z[:, p + 1], z[:, p + 2:]
        scale = torch.exp(lt[:, None] + ll)
        b = scale * eta
    else:
        b, ll, ls, lt = z[:, :p], z[:, p:2 * p], z[:, 2 * p], z[:, 2 * p + 1]
        scale = torch.exp(lt[:, None] + ll)
        eta = b / scale
    res = y - b @ X.T
    rr, w = (res ** 2).sum(1), torch.exp(-2.0 * ls)
    lam2, tau2, sig2 = torch.exp(2.0 * ll), torch.exp(2.0 * lt), torch.exp(2.0 * ls)
    half_cauchy = lambda x, x2: -math.log(math.pi) - torch.log1p(x2) + math.log(2.0) + x  # noqa: E731
    lp = (half_cauchy(ll, lam2) - 0.5 * eta ** 2 - 0.5 * LOG_2PI).sum(1)
    if not case["noncentered"]:
        lp = lp - (lt[:, None] + ll).sum(1)
    lp = lp + half_cauchy(lt, tau2) - 0.5 * sig2 - 0.5 * LOG_2PI + math.log(2.0) + ls
    lp = lp - 0.5 * rr * w - n * ls - 0.5 * n * LOG_2PI
    g = (res @ X) * w[:, None]
    shrink, top = 2.0 * lam2 / (1.0 + lam2), 2.0 * tau2 / (1.0 + tau2) - 1.0
    dls = sig2 - 1.0 - rr * w + n
    if case["noncentered"]:
        bg = b * g
        grad = torch.cat([shrink - 1.0 - bg, dls[:, None], (top - bg.sum(1))[:, None], eta - scale * g], dim=1)
    else:
        grad = torch.cat([b / scale ** 2 - g, shrink - eta ** 2, dls[:, None],
                          (top + (1.0 - eta ** 2).sum(1))[:, None]], dim=1)
    return -lp, grad


def _exact_sv(case, r, z):
    r, z = (torch.as_tensor(v, device="cuda").double() for v in (r, z))
    T = r.shape[0]
    h, lnu, ls = z[:, :T].clone(), z[:, T:T + 1], z[:, T + 1:]
    nu, s, base = torch.exp(lnu), torch.exp(ls), h
    if case["noncentered"]:
        walk = base.cumsum(1)
        h = s * walk
    y2 = (r * torch.exp(-h)) ** 2
    frac = y2 / (nu + y2)
    log1p = torch.log1p(y2 / nu)
    lp = math.log(10.0) + math.log(0.1) - 10.0 * s + ls - 0.1 * nu + lnu
    norm = 0.5 * lnu + 0.5 * math.log(math.pi) + torch.lgamma(0.5 * nu) - torch.lgamma(0.5 * (nu + 1.0))
    lp = lp - 0.5 * (nu + 1.0) * log1p.sum(1, True) - h.sum(1, True) - T * norm
    dnu = (-0.5 * log1p.sum(1, True) + 0.5 * (nu + 1.0) / nu * frac.sum(1, True) - 0.5 * T / nu
           - 0.5 * T * torch.digamma(0.5 * nu) + 0.5 * T * torch.digamma(0.5 * (nu + 1.0)) - 0.1)
    a = (nu + 1.0) * frac - 1.0
    if case["noncentered"]:
        lp = lp - 0.5 * (base ** 2).sum(1, True) - 0.5 * T * LOG_2PI
        g = base - s * a.flip(1).cumsum(1).flip(1)
        gs = -s * (a * walk).sum(1, True) + 10.0 * s - 1.0
    else:
        d = torch.diff(h, dim=1, prepend=torch.zeros_like(lnu))
        lp = lp - 0.5 * (d ** 2).sum(1, True) / s ** 2 - T * ls - 0.5 * T * LOG_2PI
        g = (d - torch.cat([d[:, 1:], torch.zeros_like(lnu)], dim=1)) / s ** 2 - a
        gs = -(d ** 2).sum(1, True) / s ** 2 + T + 10.0 * s - 1.0
    return -lp[:, 0], torch.cat([g, -(dnu * nu + 1.0), gs], dim=1)


def exact(case, seed):
    """The potential and its gradient in 64 bits.  A transition's outcome also depends on the engine's random
    numbers, so calls that sample have no such value."""
    if case["call"] != "potential":
        return None
    if case["family"] == "logreg":
        X, y, z, _ = _logreg_data(case, seed)
        return _exact_logreg(X, y, z)
    if case["family"] == "horseshoe":
        return _exact_horseshoe(case, *_horseshoe_data(case, seed))
    r, z, _ = _sv_data(case, seed)
    return _exact_sv(case, r, z)
