"""The work that users of this framework have it do, as cases that can be timed and compared.

Each case is a dict of plain values; ``prepare`` makes what a user's program has in hand before the
call (handles, batches, networks, inputs), ``run`` is one pass through the public entry points, and
``work`` says what that pass cannot do without. The sizes are those of the benchmark configurations
(arbo_gpu_fit_gb300/configs.py), of the fit (arbo_gpu_fit_gb300/fit.py) and of the tests, with odd
ones between them.

Kinds of case:

* ``sim``    one simulation handle, re-seeded by its user, initialised and run; the time series and
             the end-of-run counters are read.
* ``call``   the reference-facing call ``simulation(...)``: create, initialise, run, read, destroy.
* ``batch``  many handles stepped together with new parameters and seeds (a training set of the
             surrogate, the proposals of an MCMC iteration), their incidence series read.
* ``mcmc``   the batched MCMC driver: initial states and iterations with FP64 likelihood and acceptance.
* ``train``  the surrogate network trained over minibatches, its weights read.
* ``forward`` the surrogate network's predictions.
"""
import math

import numpy as np
import torch

from arbo_gpu_fit_gb300 import _native, configs
from arbo_gpu_fit_gb300.mcmc import MCMC, chain_batch, run_batched
from arbo_gpu_fit_gb300.simulation import Batch, Parameter, Simulation, community_sizes, simulation
from arbo_gpu_fit_gb300.surrogate import MLP

N_PARAM = len(configs.PRIOR_BOX)
SERIES = ("n_incidence", "n_infected", "one_subpop", "n_count", "m_count", "m_infected")
COUNTERS = ("n_infected_subpop", "m_infected_subpop", "m_subpop_count", "m_dead_count")


def _sim(name, humans, slots, nx, ny, strains, days, spatial=False, kind="sim"):
    return {"name": name, "kind": kind, "humans": humans, "slots": slots, "nx": nx, "ny": ny, "strains": strains,
            "days": days, "spatial": spatial}


def _batch(name, instances, humans, communities, days, uneven):
    return {"name": name, "kind": "batch", "instances": instances, "humans": humans, "communities": communities,
            "days": days, "uneven": uneven}


def _net(name, kind, hidden, layers, outputs, rows, steps):
    return {"name": name, "kind": kind, "hidden": hidden, "layers": layers, "outputs": outputs, "rows": rows,
            "steps": steps}


def listed():
    return [
        # A village over a month: the smallest call, all latency and launches.
        _sim("village_month", 2_000, 10_000, 5, 5, 4, 30),
        # The small benchmark population over its year.
        _sim("small_year", 10_000, 40_000, 10, 10, 4, 365),
        # A town with one serotype (the reference ships one) and the per-community series recorded; odd sizes.
        _sim("town_spatial", 237_411, 1_187_003, 31, 29, 1, 200, spatial=True),
        # The large benchmark population, one year of it.
        _sim("large_year", 1_000_000, 6_000_000, 50, 50, 4, 365),
        # The largest population of the batched configuration, alone, half a year.
        _sim("metropolis_half_year", 2_000_000, 12_000_000, 63, 63, 4, 182),
        # The reference-facing call of a city: handle made and freed inside, as one replicate of a script.
        _sim("city_call", 100_000, 600_000, 20, 20, 4, 365, kind="call"),
        # Training runs of the surrogate / the proposals of one MCMC iteration: many small populations.
        _batch("fit_batch", 128, 10_000, 100, 365, False),
        # The batched configuration: uneven populations and networks.
        _batch("uneven_batch", 24, 2_000_000, 4_000, 90, True),
        # The fit's chains: initial states and two iterations, 8 chains of 4 replicates, a year of data.
        {"name": "mcmc_iterations", "kind": "mcmc", "chains": 8, "replicates": 4, "humans": 10_000, "side": 10,
         "days": 365, "iterations": 3},
        # The surrogate of the fit over 8,192 simulator runs: one epoch of minibatches of 256.
        _net("surrogate_epoch", "train", 512, 4, 480, 256, 32),
        # The first stage of delayed acceptance: the surrogate at the proposals of 64 chains.
        _net("surrogate_screen", "forward", 512, 4, 480, 64, 1),
        # A wide network and large minibatches, as for a training set of the specified 200,000 runs.
        _net("wide_epoch", "train", 1024, 4, 480, 4096, 8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sim", "sim", "sim", "call", "batch", "batch", "mcmc", "train", "train", "forward"])
    if kind in ("sim", "call"):
        humans = _log_int(rng, 1_500, 2_000_000 if kind == "sim" else 200_000)
        slots = int(humans * rng.uniform(3.0, 6.0))
        side = max(2, min(63, int(math.sqrt(humans / rng.uniform(60, 400)))))
        days = max(20, min(365, int(2.0e9 / (humans + slots) * rng.uniform(0.3, 1.0))))
        return _sim("", humans, slots, side, max(2, side - rng.randrange(3)), rng.choice([1, 2, 3, 4, 4, 4]), days,
                    kind == "sim" and days <= 200 and rng.random() < 0.3, kind)
    if kind == "batch":
        if rng.random() < 0.5:
            return _batch("", _log_int(rng, 8, 128), _log_int(rng, 2_000, 10_000), rng.randrange(20, 120),
                          rng.randrange(60, 366), False)
        return _batch("", _log_int(rng, 3, 24), _log_int(rng, 100_000, 2_000_000), rng.randrange(300, 4_000),
                      rng.randrange(20, 91), True)
    if kind == "mcmc":
        return {"name": "", "kind": "mcmc", "chains": rng.randrange(2, 9), "replicates": rng.randrange(1, 5),
                "humans": _log_int(rng, 2_000, 10_000), "side": rng.randrange(4, 11),
                "days": rng.randrange(90, 366), "iterations": rng.randrange(2, 4)}
    months = rng.choice([12, 36, 60, 120])
    hidden = 16 * _log_int(rng, 4, 64)
    layers = rng.randrange(2, 5)
    if kind == "train":
        rows = 16 * _log_int(rng, 2, 256)
        return _net("", kind, hidden, layers, months * 4, rows, max(4, min(32, 32_768 // rows)))
    return _net("", kind, hidden, layers, months * 4, _log_int(rng, 3, 20_000), 1)


def _workload(case, rng):
    N, M, P = case["humans"], case["slots"], case["nx"] * case["ny"]
    sp = configs.base_param(N, M, 1)
    sp.metaPop = float(P)
    sp.nStrains = case["strains"]
    sp.recordSpatial = 1 if case["spatial"] else 0
    w = np.exp(0.8 * rng.standard_normal(P))
    return (Parameter(sp), configs.rect_network(case["nx"], case["ny"]), community_sizes(w, N), community_sizes(w, M))


def _theta(rng, n):
    lo = np.array([b[1] for b in configs.PRIOR_BOX])
    hi = np.array([b[2] for b in configs.PRIOR_BOX])
    return lo + (hi - lo) * rng.uniform(size=(n, N_PARAM))


def _weights(case, rng):
    """Uniform(+-1/sqrt(fan_in)) weights and biases of every layer, in the padded shapes of the network."""
    dims = [16] + [case["hidden"]] * case["layers"] + [case["outputs"]]
    out = []
    for l in range(len(dims) - 1):
        fan = N_PARAM if l == 0 else dims[l]
        bound = 1.0 / math.sqrt(fan)
        w = rng.uniform(-bound, bound, (dims[l + 1], dims[l])).astype(np.float32)
        if l == 0:
            w[:, N_PARAM:] = 0.0
        out.append((w, rng.uniform(-bound, bound, dims[l + 1]).astype(np.float32)))
    return out


def _data(case, rng):
    """Normalised parameter vectors and log(1 + monthly cases) that vary smoothly with them."""
    n = case["rows"] * case["steps"]
    x = rng.uniform(-1.0, 1.0, (n, N_PARAM)).astype(np.float32)
    a = rng.standard_normal((N_PARAM, case["outputs"])).astype(np.float32)
    y = (2.5 + 2.5 * np.sin(x @ a)).astype(np.float32) if case["kind"] != "forward" else None
    return x, y


def prepare(case, seed):
    _native.check(_native.load().arbo_set_device(0))
    rng = np.random.default_rng([seed, 17])
    kind = case["kind"]
    if kind in ("sim", "call"):
        par, net, ns, ms = _workload(case, rng)
        state = {"case": case, "par": par, "net": net, "ns": ns, "ms": ms, "seed": int(rng.integers(1 << 40))}
        if kind == "sim":
            state["sim"] = Simulation(par, net, ns, ms, max_time=case["days"], seed=state["seed"])
        return state
    if kind == "batch":
        if case["uneven"]:
            ws = configs.batched(case["instances"], seed=int(rng.integers(1 << 30)), max_time=case["days"],
                                 human_range=(20_000, case["humans"]), comm_range=(100, case["communities"]))
        else:
            nx, ny = configs.near_square(case["communities"])
            one = {"humans": case["humans"], "slots": 6 * case["humans"], "nx": nx, "ny": ny, "strains": 4,
                   "spatial": False}
            par, net, ns, ms = _workload(one, rng)
            w = configs.Workload("fit", par, net, ns, ms, case["days"], 1)
            ws = [w] * case["instances"]
        sims = [Simulation(w.parameter, w.network, w.n_sizes, w.m_sizes, max_time=w.max_time, seed=w.seed) for w in ws]
        th = _theta(rng, len(ws))
        return {"case": case, "sims": sims, "batch": Batch(sims) if case["uneven"] else chain_batch(sims),
                "params": [configs.apply_theta(w.parameter.simulation, t) for w, t in zip(ws, th)],
                "seeds": [int(s) for s in rng.integers(1 << 40, size=len(ws))]}
    if kind == "mcmc":
        side, N = case["side"], case["humans"]
        w = configs.scaled(N, 6 * N, side, case["days"], seed=int(rng.integers(1 << 30)))
        C, R, months = case["chains"], case["replicates"], 12
        observed = rng.poisson(rng.uniform(0.0, 0.004 * N, (months, 4))).astype(np.uint32)
        lo = np.array([b[1] for b in configs.PRIOR_BOX])
        hi = np.array([b[2] for b in configs.PRIOR_BOX])
        chains = MCMC(w, observed, C, 0.04 * (hi - lo), seed=int(rng.integers(1 << 40)), replicates=R,
                      max_iters=case["iterations"])
        sims = chains.make_sims(C * R)
        return {"case": case, "chains": chains, "sims": sims, "batch": chain_batch(sims),
                "theta0": lo + (hi - lo) * rng.uniform(0.25, 0.75, (C, N_PARAM))}
    weights = _weights(case, rng)
    x, y = _data(case, rng)
    rows = case["rows"]
    net = MLP(N_PARAM, case["hidden"], case["layers"], case["outputs"],
              max_batch=min(4096, rows + (-rows) % 16), seed=1)
    for l, (w, b) in enumerate(weights):
        net.set_layer(l, w, b)
    return {"case": case, "net": net, "x": x, "y": y}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sim":
        sim = state["sim"]
        sim.init()
        sim.run()
        out = {k: sim.series(k) for k in SERIES}
        if case["spatial"]:
            out["infected_subpop"] = sim.series("infected_subpop")
        for k in COUNTERS:
            out[k] = sim.counters(k)
        return out
    if kind == "call":
        return simulation(state["par"], state["net"], case["days"], state["ns"], state["ms"], seed=state["seed"])
    if kind == "batch":
        b = state["batch"]
        b.set_params(state["params"], state["seeds"])
        b.init()
        b.run()
        daily = [s.series("n_incidence") for s in state["sims"]]
        return np.concatenate(daily, axis=1)
    if kind == "mcmc":
        m = state["chains"]
        run_batched(m, case["iterations"], state["theta0"], state["sims"], state["batch"])
        chain, accepted = m.chain(case["iterations"])
        now = m.state()
        return {"chain": chain, "accepted": accepted, "logpost": now["logpost"], "loglik": now["loglik"]}
    net, x, y = state["net"], state["x"], state["y"]
    if kind == "forward":
        return net.forward(x)
    rows = case["rows"]
    losses = [net.train_step(x[i:i + rows], y[i:i + rows], 1e-3) for i in range(0, len(x), rows)]
    layers = [net.layer(l)[:2] for l in range(net.layers)]
    return {"losses": np.array(losses), "w": [l[0] for l in layers], "b": [l[1] for l in layers]}


def _agent_bytes(humans, slots, days):
    """Each step asks of every human and of every mosquito slot whether something is due (a 4-byte event time; a
    slot's state byte too), and writes each newborn (state, survival draw, birth and death time): about a tenth of
    the expected 4 mosquitoes per human."""
    return days * (4.0 * humans + 5.0 * slots + 14.0 * 0.4 * humans)


def work(case):
    kind = case["kind"]
    if kind in ("sim", "call"):
        out = 4.0 * (case["days"] + 1) * (4 * case["strains"] + 2)
        if case["spatial"]:
            out += 4.0 * (case["days"] + 1) * case["strains"] * case["nx"] * case["ny"]
        return {"bytes": _agent_bytes(case["humans"], case["slots"], case["days"]) + out, "flops": 0.0}
    if kind == "batch":
        # Uneven populations are log-uniform between 20,000 and `humans`.
        lo, hi = 20_000.0, float(case["humans"])
        mean = (hi - lo) / math.log(hi / lo) if case["uneven"] else hi
        one = _agent_bytes(mean, 6 * mean, case["days"]) + 16.0 * (case["days"] + 1)
        return {"bytes": case["instances"] * one, "flops": 0.0}
    if kind == "mcmc":
        one = _agent_bytes(case["humans"], 6 * case["humans"], case["days"])
        return {"bytes": case["iterations"] * case["chains"] * case["replicates"] * one, "flops": 0.0}
    dims = [16] + [case["hidden"]] * case["layers"] + [case["outputs"]]
    weights = sum(i * o for i, o in zip(dims, dims[1:]))
    n = case["rows"] * case["steps"]
    if kind == "forward":
        return {"bytes": 4.0 * (n * (N_PARAM + case["outputs"]) + weights), "flops": 2.0 * n * weights}
    # Forward, backward signal (not into the inputs) and weight gradients.
    flops = 2.0 * n * (2 * weights + weights - dims[0] * dims[1])
    per_step = 24.0 * weights  # weights and both moments, read and written
    return {"bytes": 4.0 * n * (N_PARAM + case["outputs"]) + case["steps"] * per_step, "flops": flops}


def _forward64(x, params):
    """Pre-activations and activations of every layer, in 64 bits."""
    zs, hs = [], [x]
    for l, (w, b) in enumerate(params):
        z = hs[-1] @ w.T + b
        zs.append(z)
        hs.append(z * torch.sigmoid(z) if l + 1 < len(params) else z)
    return zs, hs


def _grads64(x, y, params):
    zs, hs = _forward64(x, params)
    e = hs[-1] - y
    dz = 2.0 * e / e.numel()
    grads = [None] * len(params)
    for l in range(len(params) - 1, -1, -1):
        grads[l] = (dz.T @ hs[l], dz.sum(0))
        if l:
            s = torch.sigmoid(zs[l - 1])
            dz = (dz @ params[l][0]) * (s * (1.0 + zs[l - 1] * (1.0 - s)))
    return float((e * e).mean()), grads


def exact(case, seed):
    """The network cases in 64 bits; simulations return whole numbers, which have no rounding, and the chains' 64-bit
    numbers follow from them."""
    kind = case["kind"]
    if kind not in ("train", "forward"):
        return None
    rng = np.random.default_rng([seed, 17])
    weights = _weights(case, rng)
    x, y = _data(case, rng)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    params = [tuple(torch.from_numpy(a).to(dev).double() for a in wb) for wb in weights]
    xd = torch.zeros((len(x), 16), dtype=torch.float64, device=dev)
    xd[:, :N_PARAM] = torch.from_numpy(x).to(dev).double()
    if kind == "forward":
        return _forward64(xd, params)[1][-1].cpu().numpy()
    yd = torch.from_numpy(y).to(dev).double()
    lr, b1, b2, eps = 1e-3, 0.9, 0.999, 1e-8
    mom = [[torch.zeros_like(p) for p in wb] for wb in params]
    var = [[torch.zeros_like(p) for p in wb] for wb in params]
    losses, rows = [], case["rows"]
    for k in range(case["steps"]):
        loss, grads = _grads64(xd[k * rows:(k + 1) * rows], yd[k * rows:(k + 1) * rows], params)
        losses.append(loss)
        new = []
        for l, wb in enumerate(params):
            out = []
            for i, p in enumerate(wb):
                mom[l][i] = b1 * mom[l][i] + (1 - b1) * grads[l][i]
                var[l][i] = b2 * var[l][i] + (1 - b2) * grads[l][i] ** 2
                c1, c2 = 1 - b1 ** (k + 1), 1 - b2 ** (k + 1)
                out.append(p - lr * (mom[l][i] / c1) / (torch.sqrt(var[l][i] / c2) + eps))
            new.append(tuple(out))
        params = new
    return {"losses": np.array(losses), "w": [p[0].cpu().numpy() for p in params],
            "b": [p[1].cpu().numpy() for p in params]}
