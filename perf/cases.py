"""What a user of this framework has it do, as timed cases.

Two halves, as the package has them.  The agent-based engine: a world stepped hour by hour, a
whole run of a world (10 thousand to 4 million agents), a run from the config file on (world
build to final records), a batched ensemble of uneven worlds, and the curves of a batch of
sweep points.  The learned surrogate: one minibatch's gradients, a training call, curves for a
list of parameter points, and the screen of many candidates against a target curve.

Agent states, counts and cells are whole numbers, the same for the same config and seed on
every machine; the surrogate's outputs are computed numbers, and `exact` gives them in 64 bits.
"""
from __future__ import annotations

import json
import math

import numpy as np
import torch

from epirust_gb300 import Config, Ensemble, Epidemiology
from epirust_gb300.surrogate import Surrogate, config_for, denormalise, latin_hypercube, simulate_curves
from epirust_gb300.workloads import SMALL_POX, config_dict, ensemble_params

# a fast disease with every compartment (tests and tests/golden/fast_1m_2500.json)
FAST = {
    "regular_transmission_start_day": 1, "high_transmission_start_day": 3, "last_day": 6,
    "asymptomatic_last_day": 9, "mild_infected_last_day": 12,
    "regular_transmission_rate": 0.3, "high_transmission_rate": 0.6, "death_rate": 0.3,
    "percentage_asymptomatic_population": 0.3, "percentage_severe_infected_population": 0.4,
    "exposed_duration": 12, "pre_symptomatic_duration": 10,
}


def listed() -> list:
    return [
        # An interactive driver of a small town: simulate(hour) and process_interventions(counts)
        # hour by hour, as the reference's own loop does, then the citizens' records.  Single
        # hours of 10,000 agents: launches and waits are all there is.
        {"name": "step_10k", "kind": "step", "agents": 10_000, "grid": 250, "hours": 48, "disease": "small_pox",
         "interventions": "none", "exposed": 5},
        # The reference's default world (10,000 agents, 250 grid, 100 days) run again and again
        # from the same start, with its final records: a long chain of short launches.
        {"name": "run_10k", "kind": "run", "agents": 10_000, "grid": 250, "hours": 2400, "disease": "small_pox",
         "interventions": "none", "exposed": 50},
        # The command line's work: config in, engine built, a run with a lockdown and a
        # vaccination, records out, engine gone.  Odd sizes, everything for the first time.
        {"name": "cold_98k", "kind": "cold", "agents": 97_531, "grid": 787, "hours": 1200, "disease": "fast",
         "interventions": "all", "exposed": 31},
        # The benchmark's city: 1M agents on 2,500 x 2,500, 200 days, lockdown, vaccination and
        # hospital build.
        {"name": "run_1m", "kind": "run", "agents": 1_000_000, "grid": 2500, "hours": 4800, "disease": "small_pox",
         "interventions": "all", "exposed": 50},
        # A large city whose working set (about 350 MB) does not fit the L2.
        {"name": "run_4m", "kind": "run", "agents": 4_000_000, "grid": 5000, "hours": 1200, "disease": "small_pox",
         "interventions": "none", "exposed": 2000},
        # Many uneven worlds at once (10,000 to 500,000 agents, rates and seeds their own): ten
        # days of the 256-replicate ensemble.
        {"name": "ensemble_256", "kind": "ensemble", "replicates": 256, "n_min": 1e4, "n_max": 5e5, "hours": 241},
        # A batch of sweep points as the surrogate's training data is made: worlds of one size,
        # a lockdown and a vaccination each, created, run and reduced to daily curves.
        {"name": "curves_64", "kind": "curves", "points": 64, "agents": 50_000, "grid": 560, "days": 25},
        # One minibatch's loss and gradients of one network: the latency of a forward and a
        # backward pass.
        {"name": "gradients_1", "kind": "gradients", "hidden": 512, "layers": 3, "days": 100, "in_dim": 8, "batch": 256,
         "members": 1},
        # Fine-tuning one network from given weights: weights in, 100 Adam steps, weights out.
        {"name": "train_1", "kind": "train", "hidden": 512, "layers": 3, "days": 100, "in_dim": 8, "batch": 256,
         "members": 1, "samples": 4096, "steps": 100},
        # The sweep's ensemble of five, trained together.
        {"name": "train_5", "kind": "train", "hidden": 512, "layers": 3, "days": 100, "in_dim": 8, "batch": 256,
         "members": 5, "samples": 3584, "steps": 100},
        # Five members' curves for the points a sweep keeps (an odd number of them).
        {"name": "predict_1k", "kind": "predict", "hidden": 512, "layers": 3, "days": 100, "in_dim": 8, "members": 5,
         "points": 1003},
        # The screen: 65,536 candidates scored by five members against one target curve.
        {"name": "score_64k", "kind": "score", "hidden": 512, "layers": 3, "days": 100, "in_dim": 8, "members": 5,
         "points": 65_536},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["step", "run", "run", "cold", "ensemble", "curves", "gradients", "train", "predict", "score"])
    if kind in ("step", "run", "cold"):
        n = _log(rng, 3_000, {"step": 100_000, "run": 3_000_000, "cold": 500_000}[kind])
        density = rng.uniform(0.06, 0.3)
        most = {"step": 96, "run": min(4800, int(2.4e9 / n)), "cold": min(2400, int(1e9 / n))}[kind]
        disease = rng.choice(["small_pox", "fast"])
        return {"kind": kind, "agents": n, "grid": int(math.ceil(math.sqrt(n / density))),
                "hours": _log(rng, 24 if kind == "step" else 100, max(most, 101)), "disease": disease,
                "interventions": "none" if kind == "step" else rng.choice(["none", "all"]),
                "exposed": max(10, int(n * rng.uniform(2e-4, 2e-3)))}
    if kind == "ensemble":
        return {"kind": kind, "replicates": _log(rng, 4, 192), "n_min": 3e3, "n_max": float(_log(rng, 1e4, 3e5)),
                "hours": rng.randrange(30, 241)}
    if kind == "curves":
        n = _log(rng, 5_000, 100_000)
        return {"kind": kind, "points": _log(rng, 3, 64), "agents": n, "grid": int(math.ceil(math.sqrt(n / 0.16))),
                "days": rng.randrange(5, 26)}
    net = {"kind": kind, "hidden": rng.choice([128, 256, 384, 512]), "layers": rng.randrange(1, 5),
           "days": rng.randrange(7, 110), "in_dim": rng.randrange(3, 17), "members": rng.randrange(1, 6)}
    if kind in ("gradients", "train"):
        net["batch"] = rng.choice([128, 256, 512])
    if kind == "train":
        net.update(samples=_log(rng, 600, 4096), steps=_log(rng, 8, 100))
    if kind in ("predict", "score"):
        net["points"] = _log(rng, 1, 4096 if kind == "predict" else 65_536)
    return net


# ---------------------------------------------------------------- the engine
def _seed(seed: int) -> int:
    return (0x9E3779B97F4A7C15 * (seed + 1) >> 3) & (2 ** 63 - 1)


def _world(case: dict, seed: int) -> str:
    n = case["agents"]
    interventions, extra = [], {}
    if case["interventions"] == "all":  # thresholds and hours in the benchmark's proportions
        interventions = [
            {"Lockdown": {"at_number_of_infections": max(20, n // 1000), "essential_workers_population": 0.1}},
            {"Vaccinate": {"at_hour": case["hours"] // 2, "percent": 0.2}},
        ]
        extra["hospital_occupancy_trigger"] = 0.7
    disease = SMALL_POX if case["disease"] == "small_pox" else FAST
    return json.dumps(config_dict(n, case["grid"], case["hours"], _seed(seed), disease, exposed=case["exposed"],
                                  interventions=interventions, **extra))


def _points(case: dict, seed: int) -> list:
    """Sweep points as engine configs."""
    hours = 24 * case["days"] + 1
    return [config_for(d, case["agents"], case["grid"], hours, seed=_seed(seed) // 7 + i, per_agents=100_000)
            for i, d in enumerate(denormalise(latin_hypercube(case["points"], 8, seed)))]


def _words(a: np.ndarray) -> np.ndarray:
    """Counts rows or citizen records as the 32-bit words and bytes they are."""
    if a.dtype.itemsize == 28:
        return a.view(np.uint32).reshape(len(a), 7)
    return a.view(np.uint8).reshape(len(a), a.dtype.itemsize)


# ---------------------------------------------------------------- the surrogate
def _shapes(case: dict) -> list:
    h = case["hidden"]
    return [(h, case["in_dim"])] + [(h, h)] * (case["layers"] - 1) + [(6 * case["days"], h)]


def _weights(case: dict, seed: int) -> np.ndarray:
    """(members, parameters): torch.nn.Linear's uniform draw, W then b, layer by layer."""
    rng = np.random.default_rng([seed, 1])
    flat = []
    for _ in range(case["members"]):
        for n, k in _shapes(case):
            bound = 1.0 / math.sqrt(k)
            flat += [rng.uniform(-bound, bound, n * k), rng.uniform(-bound, bound, n)]
    return np.concatenate(flat).astype(np.float32).reshape(case["members"], -1)


def _curves(case: dict, u: np.ndarray, seed: int) -> np.ndarray:
    """Smooth standardised curves of the points u, as epidemics' daily compartments are."""
    rng = np.random.default_rng([seed, 2])
    t = np.arange(case["days"]) / case["days"]
    out = []
    for _ in range(6):
        a, b, c = (u @ rng.normal(size=(case["in_dim"], 3))).T
        out.append(np.tanh(a[:, None] + 4.0 * (t[None, :] - 0.5) * (1.0 + b[:, None] ** 2)) + 0.3 * c[:, None] * t[None, :])
    return np.concatenate(out, axis=1).astype(np.float32)


def _net_inputs(case: dict, seed: int) -> dict:
    rng = np.random.default_rng([seed, 3])
    rows = {"gradients": case.get("batch"), "train": case.get("samples")}.get(case["kind"], case.get("points"))
    x = rng.random((rows, case["in_dim"])).astype(np.float32)
    data = {"x": x, "w": _weights(case, seed)}
    if case["kind"] in ("gradients", "train"):
        data["y"] = _curves(case, x, seed)
    if case["kind"] == "score":
        data["target"] = _curves(case, rng.random((1, case["in_dim"])).astype(np.float32), seed)[0]
    return data


# ---------------------------------------------------------------- prepare and run
def prepare(case: dict, seed: int) -> dict:
    state = dict(case)
    kind = case["kind"]
    if kind in ("step", "run"):
        state["engine"] = Epidemiology(Config(_world(case, seed)))
        state["engine"].save_state()
    elif kind == "cold":
        state["config"] = _world(case, seed)
    elif kind == "ensemble":
        params = ensemble_params(replicates=case["replicates"], seed=seed + 11, hours=case["hours"], n_min=case["n_min"],
                                 n_max=case["n_max"])
        state["engine"] = Ensemble(params)
        state["engine"].save_state()
    elif kind == "curves":
        state["configs"] = _points(case, seed)
    else:
        data = _net_inputs(case, seed)
        net = Surrogate(in_dim=case["in_dim"], out_dim=6 * case["days"], hidden=case["hidden"],
                        hidden_layers=case["layers"], batch=case.get("batch", 256), seed=seed, members=case["members"])
        net.set_params(data["w"])
        if kind == "train":
            net.set_dataset(data["x"], data["y"])
        state.update(data, net=net, shuffle=seed + 5)
    return state


def run(state: dict):
    kind = state["kind"]
    if kind == "step":
        eng = state["engine"]
        eng.restore_state()
        rows = []
        for hour in range(1, state["hours"] + 1):
            c = eng.simulate(hour)
            eng.process_interventions(c)
            rows.append((c.hour, c.susceptible, c.exposed, c.infected, c.hospitalized, c.recovered, c.deceased))
        return [np.array(rows, dtype=np.uint32), _words(eng.snapshot())]
    if kind == "run":
        eng = state["engine"]
        eng.restore_state()
        return [_words(eng.run()), _words(eng.snapshot())]
    if kind == "cold":
        with Epidemiology(Config(state["config"])) as eng:
            return [_words(eng.run()), _words(eng.snapshot())]
    if kind == "ensemble":
        state["engine"].restore_state()
        rows = state["engine"].run()
        return [np.array([len(r) for r in rows], dtype=np.int64), _words(np.concatenate(rows))]
    if kind == "curves":
        return simulate_curves(state["configs"], state["days"])
    net = state["net"]
    if kind == "gradients":
        loss, grads = net.gradients(state["x"], state["y"])
        return [np.atleast_1d(np.asarray(loss, dtype=np.float32)), np.atleast_2d(grads)]
    if kind == "train":
        net.set_params(state["w"])
        losses = net.train(state["steps"], seed=state["shuffle"])
        return [np.atleast_2d(losses), np.atleast_2d(net.get_params())]
    if kind == "predict":
        return net.predict_members(state["x"])
    return net.score_members(state["x"], state["target"])


# ---------------------------------------------------------------- what a pass cannot do without
def _world_bytes(n: float, grid: float, hours: int) -> float:
    """A day of a world: in the 16 hours of 7..22 each agent's position, state, house and office
    are read (20 B) and its position written (4 B), and one bit per cell read and written; at
    hours 0 and 23 the state is read, and hour 1 reads and writes its first word."""
    cells = (grid + 1.0) ** 2
    day = 16.0 * (24.0 * n + cells / 4.0) + 2.0 * 8.0 * n + 8.0 * n
    return day * hours / 24.0


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("step", "run", "cold"):
        n = case["agents"]
        hours = case["hours"] - (kind != "step")
        return {"bytes": _world_bytes(n, case["grid"], hours) + 56.0 * n + 28.0 * hours, "flops": 0.0}
    if kind == "ensemble":  # populations are log-uniform: their mean stands for the draw
        lo, hi = case["n_min"], case["n_max"]
        n = (hi - lo) / math.log(hi / lo)
        return {"bytes": case["replicates"] * _world_bytes(n, math.sqrt(n / 0.16), case["hours"] - 1), "flops": 0.0}
    if kind == "curves":
        return {"bytes": case["points"] * (_world_bytes(case["agents"], case["grid"], 24 * case["days"]) + 24.0 * case["days"]),
                "flops": 0.0}
    params = sum(n * k + n for n, k in _shapes(case))
    macs = sum(n * k for n, k in _shapes(case))
    out = 6 * case["days"]
    e = case["members"]
    if kind == "gradients":
        b = case["batch"]
        return {"bytes": 4.0 * (b * (case["in_dim"] + out) + 2.0 * e * params), "flops": 6.0 * e * b * macs}
    if kind == "train":
        b, s = case["batch"], case["steps"]
        # weights, two moments read and written, a minibatch read, each step
        return {"bytes": 4.0 * e * s * (6.0 * params + b * (case["in_dim"] + out)), "flops": 6.0 * e * s * b * macs}
    p = case["points"]
    written = e * p * (out if kind == "predict" else 1)
    return {"bytes": 4.0 * (e * params + p * case["in_dim"] + written), "flops": 2.0 * e * p * macs}


# ---------------------------------------------------------------- the values in 64 bits
def _split(case: dict, flat: torch.Tensor) -> list:
    """(members, parameters) -> [(W, b)] with a leading member axis."""
    out, o = [], 0
    for n, k in _shapes(case):
        w = flat[:, o:o + n * k].reshape(-1, n, k)
        b = flat[:, o + n * k:o + n * k + n].reshape(-1, 1, n)
        out.append((w, b))
        o += n * k + n
    return out


def _forward(case: dict, flat: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    h = x
    layers = _split(case, flat)
    for l, (w, b) in enumerate(layers):
        h = h @ w.transpose(1, 2) + b
        if l + 1 < len(layers):
            h = torch.nn.functional.gelu(h)
    return h


def _batches(case: dict, seed: int) -> np.ndarray:
    """(members, steps, batch) sample indices: member m's stream is splitmix64 from seed + m, a
    Fisher-Yates permutation each epoch, whole minibatches only."""
    n, b, steps = case["samples"], case["batch"], case["steps"]
    mask = (1 << 64) - 1
    out = np.zeros((case["members"], steps, b), dtype=np.int64)
    for m in range(case["members"]):
        s = (seed + m) & mask
        perm = None
        for step in range(steps):
            k = step % (n // b)
            if k == 0:
                perm = list(range(n))
                for i in range(n - 1, 0, -1):
                    s = (s + 0x9E3779B97F4A7C15) & mask
                    z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
                    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
                    j = (z ^ (z >> 31)) % (i + 1)
                    perm[i], perm[j] = perm[j], perm[i]
            out[m, step] = perm[k * b:(k + 1) * b]
    return out


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind not in ("gradients", "train", "predict", "score"):
        return None  # whole numbers, and curves that are their quotients
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    data = {k: torch.from_numpy(v).to(dev, torch.float64) for k, v in _net_inputs(case, seed).items()}
    flat, x = data["w"], data["x"]
    if kind == "predict":
        return _forward(case, flat, x[None]).cpu().numpy()
    if kind == "score":
        parts = [((_forward(case, flat, x[None, i:i + 4096]) - data["target"]) ** 2).sum(dim=2)
                 for i in range(0, len(x), 4096)]
        return torch.cat(parts, dim=1).cpu().numpy()
    flat = flat.clone().requires_grad_(True)
    if kind == "gradients":
        loss = ((_forward(case, flat, x[None]) - data["y"]) ** 2).mean(dim=(1, 2))
        (g,) = torch.autograd.grad(loss.sum(), flat)
        return [loss.detach().cpu().numpy(), g.cpu().numpy()]
    m, v = torch.zeros_like(flat), torch.zeros_like(flat)
    losses = []
    idx = torch.from_numpy(_batches(case, seed + 5)).to(dev)
    for t in range(1, case["steps"] + 1):
        pick = idx[:, t - 1]
        loss = ((_forward(case, flat, x[pick]) - data["y"][pick]) ** 2).mean(dim=(1, 2))
        (g,) = torch.autograd.grad(loss.sum(), flat)
        losses.append(loss.detach())
        with torch.no_grad():  # Adam (Kingma & Ba 2015) with the handle's defaults
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            flat = flat - 1e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
        flat.requires_grad_(True)
    return [torch.stack(losses, dim=1).cpu().numpy(), flat.detach().cpu().numpy()]
