"""The work that users of the engine have it do, as measurable cases.

Every case is a dict of plain values; `kind` names the entry point it goes
through:

  one         FixedFacoGpu.run_iterations: one instance, one colony
  session     GpuSession.solve: a fixed panel with the default settings
  panel       FacoBatchEngine.begin / step / finish: (instance, seed) colonies
  population  FacoBatchEngine.evaluate_population_evaluations: GP controllers
  prior       a stepwise panel under the learned edge prior, refreshed between
              steps, with the training rows read at its end
  score       score_cuda: GP programs over a block of colony features
  train       prior.train: Adam epochs of the edge-prior network
  pheromone   faco_pheromone_step_noalloc on device buffers

Sizes and settings are those of the benchmark's and the experiments'
workloads, of the session's and the settings' defaults, and odd ones between.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import gplsaco_gb300 as g
from gplsaco_gb300 import _lib, instances, prior
from gplsaco_gb300.programs import random_program


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _panel(name, n, count, seeds, ants, k, w, ls_mode, mne, iterations, clustered):
    c = {"kind": "panel", "n_lo": n[0], "n_hi": n[1], "instances": count, "seeds": seeds, "ants": ants, "k": k,
         "w": w, "ls_mode": ls_mode, "mne": mne, "retention": 0.98, "iterations": iterations, "clustered": clustered}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a single small instance solved interactively: one colony, the
        # default ant count (64), a short budget -- launches and latency
        {"name": "one_n100", "kind": "one", "n": 100, "iterations": 64, "mne": 8, "clustered": False},
        # the resident session's panel with every default: 32 colonies, the
        # ant-count rule (128 ants at this size), an odd instance size
        {"name": "session_n537", "kind": "session", "n": 537, "colonies": 32, "instances": 8, "mne": 8,
         "iterations": 100, "clustered": True},
        # the throughput panel: 16 instances x 16 seeds, more ant warps than
        # the GPU holds at once, from the initial tours
        _panel("panel_n1000", (1000, 1000), 16, 16, 32, 16, 20, 0, 8, 320, False),
        # the time-to-gap runs: two sizes, two seeds per instance, few new
        # edges per ant, long enough that the colonies converge
        _panel("long_n1000_2000", (1000, 2000), 64, 2, 32, 20, 20, 0, 5, 640, True),
        # the uneven batch: every instance of another size, few ants
        _panel("uneven_n200_1000", (200, 1000), 256, 1, 16, 16, 20, 0, 8, 400, True),
        # the large clustered panel with 2-opt + Or-opt
        _panel("large_n5000_10000", (5000, 10000), 16, 5, 64, 32, 32, 1, 8, 80, True),
        # one generation of GP controllers, the engine's own features
        {"name": "population_spec3", "kind": "population", "n": 500, "programs": 128, "panel": 1, "ants": 32,
         "spec": 3, "iterations": 250, "clustered": False},
        # one generation of GP controllers, the reference's 12 features
        {"name": "population_spec2", "kind": "population", "n": 500, "programs": 128, "panel": 1, "ants": 32,
         "spec": 2, "iterations": 250, "clustered": False},
        # the learned prior on half of a panel's colonies, refreshed as the
        # trails move, then the rows that a next training round reads
        {"name": "prior_n1000_2000", "kind": "prior", "n_lo": 1000, "n_hi": 2000, "instances": 16, "seeds": 2,
         "ants": 32, "k": 20, "w": 20, "mne": 6, "iterations": 64, "refresh": 10, "gamma": 2, "clustered": True},
        # scoring a whole population's actions outside the loop
        {"name": "score_4096", "kind": "score", "programs": 128, "colonies": 4096},
        # training the prior's network on rows of earlier runs
        {"name": "train_240k", "kind": "train", "rows": 240_000, "batch": 8192, "epochs": 6},
        # the trail update of a caller that holds its own device memory
        {"name": "pheromone_n5915", "kind": "pheromone", "n": 5915, "k": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["one", "session", "panel", "panel", "panel", "population", "prior", "score", "train",
                       "pheromone"])
    if kind == "one":
        return {"kind": kind, "n": _log(rng, 50, 2000), "iterations": _log(rng, 16, 100),
                "mne": rng.choice([4, 8, 12]), "clustered": rng.random() < 0.5}
    if kind == "session":
        return {"kind": kind, "n": _log(rng, 100, 1500), "colonies": rng.choice([8, 16, 32]),
                "instances": rng.randint(1, 8), "mne": rng.choice([4, 8]), "iterations": _log(rng, 20, 100),
                "clustered": rng.random() < 0.5}
    if kind == "panel":
        hi = _log(rng, 200, 10000)
        lo = hi if rng.random() < 0.4 else int(hi * rng.uniform(0.2, 1.0))
        count, seeds = rng.randint(1, 16), rng.randint(1, 16)
        ants = rng.choice([8, 16, 31, 32, 64])
        # no more node visits than the largest listed panel's
        most = 16 * 5 * 64 * 7500 * 80 / (count * seeds * ants * hi)
        oropt = int(rng.random() < 0.35)
        return _panel("", (lo, hi), count, seeds, ants, rng.choice([8, 15, 16, 20, 32]), rng.choice([10, 20, 27, 32]),
                      oropt, rng.randint(3, 12), max(8, min(int(most), _log(rng, 16, 400))), rng.random() < 0.6)
    if kind == "population":
        return {"kind": kind, "n": _log(rng, 100, 1000), "programs": rng.randint(3, 64), "panel": rng.randint(1, 3),
                "ants": rng.choice([16, 32]), "spec": rng.choice([2, 3]), "iterations": _log(rng, 30, 200),
                "clustered": rng.random() < 0.5}
    if kind == "prior":
        hi = _log(rng, 300, 2500)
        return {"kind": kind, "n_lo": int(hi * rng.uniform(0.4, 1.0)), "n_hi": hi, "instances": rng.randint(2, 16),
                "seeds": rng.randint(1, 3), "ants": rng.choice([16, 32]), "k": rng.choice([16, 20, 32]), "w": 20,
                "mne": rng.randint(4, 8), "iterations": _log(rng, 20, 80), "refresh": rng.randint(5, 20),
                "gamma": rng.choice([1, 2]), "clustered": rng.random() < 0.7}
    if kind == "score":
        programs = rng.randint(1, 128)
        return {"kind": kind, "programs": programs, "colonies": programs * rng.randint(1, max(1, 4096 // programs))}
    if kind == "train":
        return {"kind": kind, "rows": _log(rng, 5_000, 300_000), "batch": rng.choice([2048, 5000, 8192]),
                "epochs": rng.randint(1, 5)}
    return {"kind": kind, "n": _log(rng, 100, 65535), "k": rng.choice([7, 8, 10, 16, 20, 32])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _xy(n, seed, clustered):
    xy = instances.clustered(n, seed) if clustered else instances.uniform(n, seed)
    return np.ascontiguousarray(xy, dtype=np.float64)


def _instances(case, rng):
    """`instances` coordinate arrays; their sizes, uniform in [n_lo, n_hi], belong to the case."""
    sizes = np.random.default_rng([case["n_lo"], case["n_hi"]]).integers(case["n_lo"], case["n_hi"] + 1,
                                                                        case["instances"])
    return [_xy(int(n), int(rng.integers(1 << 30)), case["clustered"]) for n in sizes]


def _programs(case, rng):
    spec = case["spec"]
    return [random_program(rng, extended=True, features=10 if spec == 3 else 12, feature_spec_id=spec)
            for _ in range(case["programs"])]


def _engine(case, xys, colonies, **settings):
    engine = g.FacoBatchEngine(max(len(xy) for xy in xys), colonies, g.FixedFacoSettings(**settings))
    for i, xy in enumerate(xys):
        engine.register_problem(1 + i, xy)
    return engine


def _edge_rows(rows, rng):
    """Feature rows as candidate edges have them (lengths falling off with rank, most edges off the best
    tour) and labels that follow the geometry."""
    x = rng.random((rows, 8), dtype=np.float32)
    rank = rng.integers(0, 20, rows).astype(np.float32) / 19
    x[:, 1] = rank
    x[:, 0] = np.minimum(1.0, (0.06 + 0.3 * rank) * (0.5 + x[:, 0]))
    x[:, 3] = np.minimum(1.0, (0.2 + 0.8 * rank) * (0.6 + 0.5 * x[:, 3]))
    x[:, 4] = np.where(x[:, 4] < 0.8, 0.0, x[:, 4])
    x[:, 6] = np.where(x[:, 6] < 0.3, 1.0, np.minimum(1.0, rank * (0.5 + x[:, 6])))
    x[:, 7] = np.minimum(1.0, x[:, 7] * rank)
    y = (rng.random(rows) < 0.75 * np.exp(-7.0 * x[:, 7] - 3.0 * rank)).astype(np.float32)
    x[:, 5] = np.where(rng.random(rows) < 0.9, y, 0.0)
    return prior.to_bf16_bits(x), y


def prepare(case, seed):
    rng = np.random.default_rng([seed, 17])
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "one":
        s["solver"] = g.FixedFacoGpu(_xy(case["n"], int(rng.integers(1 << 30)), case["clustered"]), 1 + seed % 1000,
                                     g.FixedFacoSettings(retention=0.98))
        s["seed"] = int(rng.integers(1 << 40))
    elif kind == "session":
        from gplsaco_gb300.session import Instance
        s["session"] = g.GpuSession(colonies=case["colonies"])
        s["problems"] = {f"p{i}": Instance(i + 1, _xy(case["n"], int(rng.integers(1 << 30)), case["clustered"]))
                         for i in range(case["instances"])}
        s["pairs"] = [(f"p{c % case['instances']}", int(rng.integers(1 << 40))) for c in range(case["colonies"])]
        # the session registers an instance at its first solve
        s["session"].solve(s["problems"], s["pairs"], 1, {"uniform_mne": case["mne"]})
    elif kind in ("panel", "prior"):
        xys = _instances(case, rng)
        colonies = case["instances"] * case["seeds"]
        s["engine"] = _engine(case, xys, colonies, ants=case["ants"], primary_width=case["k"], ls_width=case["w"],
                              retention=case.get("retention", 0.98), ls_mode=case.get("ls_mode", 0))
        s["keys"] = np.repeat(np.arange(1, len(xys) + 1, dtype=np.uint64), case["seeds"])
        s["seeds"] = rng.integers(1 << 40, size=colonies).astype(np.uint64)
        if kind == "prior":
            s["params"] = prior.init_params(seed)
            s["enabled"] = np.tile(np.array([0, 1], np.uint8), colonies)[:colonies]
    elif kind == "population":
        xys = [_xy(case["n"], int(rng.integers(1 << 30)), case["clustered"]) for _ in range(case["panel"])]
        s["engine"] = g.FacoBatchEngine(case["n"], case["panel"],
                                        g.FixedFacoSettings(ants=case["ants"], retention=0.98),
                                        population_size=case["programs"])
        for i, xy in enumerate(xys):
            s["engine"].register_problem(1 + i, xy)
        s["keys"] = np.arange(1, case["panel"] + 1, dtype=np.uint64)
        s["seeds"] = rng.integers(1 << 40, size=case["panel"]).astype(np.uint64)
        s["programs"] = _programs(case, rng)
    elif kind == "score":
        s["programs"] = [random_program(rng, extended=True) for _ in range(case["programs"])]
        s["features"] = rng.random((12, case["colonies"], 32), dtype=np.float32)
        masks = rng.integers(1, 1 << 32, case["colonies"], dtype=np.uint64).astype(np.uint32)
        s["masks"] = np.where(rng.random(case["colonies"]) < 0.7, np.uint32(0xFFFFFFFF), masks).astype(np.uint32)
    elif kind == "train":
        s["x"], s["y"] = _edge_rows(case["rows"], rng)
        s["params"] = prior.init_params(seed % (1 << 31))
        s["seed"] = seed % (1 << 31)
    elif kind == "pheromone":
        n, k = case["n"], case["k"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        dev = {"device": "cuda", "generator": gen}
        s["parent"] = torch.randperm(n, **dev).to(torch.int32)
        # candidate rows near a node's own index, the parent's successor often among them
        offset = torch.randint(1, max(2, min(n - 1, 4 * k)), (n, k), **dev)
        s["primary"] = ((torch.arange(n, device="cuda")[:, None] + offset) % n).to(torch.int32)
        following = torch.empty(n, dtype=torch.int32, device="cuda")
        following[s["parent"].long()] = torch.roll(s["parent"], -1)
        s["primary"][:, 0] = following
        s["eta"] = 1.0 / torch.randint(1, 10**5, (n, k), **dev).float()
        s["trails"] = 1e-7 + 1.9e-6 * torch.rand((n, k), **dev)
        s["products"] = torch.zeros_like(s["trails"])
        s["lib"] = _lib.load()
        torch.cuda.synchronize()
    else:
        raise ValueError(f"unknown kind {kind}")
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
RETENTION, TAU_MIN, TAU_MAX, DEPOSIT = (float(np.float32(v)) for v in (0.98, 1e-7, 2e-6, 1.3e-8))
LEARNING_RATE = 3e-3


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "one":
        r = s["solver"].run_iterations(s["seed"], case["iterations"], case["mne"])
        return {"tour": np.array(r["tour"]), "cost": r["cost"], "steps": r["construction_steps"],
                "evaluations": r["ls_evaluations"]}
    if kind == "session":
        r, _ = s["session"].solve(s["problems"], s["pairs"], case["iterations"], {"uniform_mne": case["mne"]})
        return {"tours": np.array([it["tour"] for it in r["items"]]), "costs": np.array([it["cost"] for it in r["items"]]),
                "work": r["colony_work"].astype(np.int64)}
    if kind == "panel":
        e = s["engine"]
        e.begin(s["keys"], s["seeds"], case["mne"])
        e.step(case["iterations"])
        r = e.finish()
        return {"tours": np.concatenate(r["tours"]).astype(np.int64), "costs": r["costs"],
                "work": r["colony_work"].astype(np.int64)}
    if kind == "population":
        e = s["engine"]
        rows = e.evaluate_population_evaluations(s["keys"], s["seeds"], e.ants * case["iterations"], s["programs"])
        fields = rows[0]["control_states"][0].keys()
        return {"costs": np.array([[it["cost"] for it in r["items"]] for r in rows]),
                "tours": np.array([[it["tour"] for it in r["items"]] for r in rows]),
                "work": np.array([r["colony_work"] for r in rows]).astype(np.int64),
                "states": {f: np.array([[c[f] for c in r["control_states"]] for r in rows]) for f in fields}}
    if kind == "prior":
        e = s["engine"]
        e.begin(s["keys"], s["seeds"], case["mne"])
        e.prior_set(s["params"], s["enabled"], 0.05, case["gamma"])
        done = 0
        while done < case["iterations"]:
            steps = min(case["refresh"], case["iterations"] - done)
            e.step(steps)
            done += steps
            if done < case["iterations"]:
                e.prior_refresh()
        x, y = e.edge_data()
        rows = e.colony_rows(min(1, s["keys"].size - 1))
        r = e.finish()
        return {"x": x.astype(np.int32), "y": y, "rows": rows, "tours": np.concatenate(r["tours"]).astype(np.int64),
                "costs": r["costs"], "work": r["colony_work"].astype(np.int64)}
    if kind == "score":
        return g.score_cuda(s["programs"], s["features"], s["masks"])
    if kind == "train":
        params, losses = prior.train(s["params"], s["x"], s["y"], epochs=case["epochs"], batch=case["batch"],
                                     lr=LEARNING_RATE, seed=s["seed"])
        return {"params": params, "losses": losses}
    _lib.check(s["lib"].faco_pheromone_step_noalloc(
        case["n"], case["k"], s["primary"].data_ptr(), s["parent"].data_ptr(), RETENTION, TAU_MIN, TAU_MAX, DEPOSIT,
        s["eta"].data_ptr(), s["trails"].data_ptr(), s["products"].data_ptr(),
        torch.cuda.current_stream().cuda_stream or None))
    return {"trails": s["trails"], "products": s["products"]}


# ---------------------------------------------------------------------------
# The least that a pass has to move and compute
# ---------------------------------------------------------------------------
MLP_FLOPS = 2 * (8 * 64 + 64 * 64 + 64)     # forward pass of one row


def _colony_bytes(n, k, ants):
    """One iteration of one colony: trails read and written, heuristic read, products written; per ant the
    parent tour read and its own tour written (16-bit nodes)."""
    return 16 * n * k + 4 * n * ants


def work(case):
    kind = case["kind"]
    if kind == "one":
        return {"bytes": case["iterations"] * _colony_bytes(case["n"], 16, g.faco_ants(case["n"])), "flops": 0}
    if kind == "session":
        return {"bytes": case["iterations"] * case["colonies"] * _colony_bytes(case["n"], 16, g.faco_ants(case["n"])),
                "flops": 0}
    if kind in ("panel", "prior"):
        n, colonies = (case["n_lo"] + case["n_hi"]) / 2, case["instances"] * case["seeds"]
        total = case["iterations"] * colonies * _colony_bytes(n, case["k"], case["ants"])
        if kind == "panel":
            return {"bytes": total, "flops": 0}
        applied = -(-case["iterations"] // case["refresh"])
        rows = colonies * n * case["k"]
        return {"bytes": total + rows * (12 * applied + 20), "flops": applied * rows / 2 * MLP_FLOPS}
    if kind == "population":
        return {"bytes": case["iterations"] * case["programs"] * case["panel"] *
                _colony_bytes(case["n"], 16, case["ants"]), "flops": 0}
    if kind == "score":
        return {"bytes": case["colonies"] * (12 * 32 * 4 + 4 + 32 * 4 + 4), "flops": case["colonies"] * 32 * 20}
    if kind == "train":
        rows = case["rows"] * case["epochs"]
        return {"bytes": case["rows"] * 20, "flops": rows * 3 * MLP_FLOPS}
    return {"bytes": case["n"] * (20 * case["k"] + 4), "flops": case["n"] * case["k"] * 3}


# ---------------------------------------------------------------------------
# The same results in 64 bits, where outputs are computed numbers
# ---------------------------------------------------------------------------
def _score_exact(programs, features):
    f = features.astype(np.float64)
    colonies = f.shape[1]
    per = colonies // len(programs)
    out = np.zeros((colonies, 32))
    for i, p in enumerate(programs):
        block = f[:, i * per:(i + 1) * per]
        consts = np.array(p["constant_bits"], np.uint32).view(np.float32).astype(np.float64)
        stack = []
        for op, arg in zip(p["opcode"], p["operand"]):
            if op == 0:
                stack.append(block[arg])
                continue
            if op == 1:
                stack.append(np.full((per, 32), consts[arg]))
                continue
            t = stack.pop() if op == 10 else None
            r = stack.pop() if op != 7 else None
            x = stack.pop()
            if op == 2:
                v = x + r
            elif op == 3:
                v = x - r
            elif op == 4:
                v = x * r
            elif op == 5:
                v = np.minimum(x, r)
            elif op == 6:
                v = np.maximum(x, r)
            elif op == 7:
                v = np.abs(x)
            elif op == 8:
                v = x / np.sqrt(1.0 + r * r)
            elif op == 9:
                small = np.abs(r) < 1e-6
                v = np.where(small, 1.0, x / np.where(small, 1.0, r))
            else:
                v = np.where(x > 0.0, r, t)
            stack.append(np.clip(v, -8.0, 8.0))
        out[i * per:(i + 1) * per] = stack[0]
    return out


def _train_exact(params, x_bits, y, epochs, batch, seed):
    order = np.random.default_rng(seed).permutation(y.size)
    x = torch.from_numpy(prior.from_bf16_bits(x_bits)[order].astype(np.float64)).cuda()
    t = torch.from_numpy(y[order].astype(np.float64)).cuda()
    p = torch.from_numpy(params.astype(np.float64)).cuda()
    sizes = [64 * 8, 64, 64 * 64, 64, 64, 1]
    ends = np.cumsum(sizes)
    m, v, step, losses = torch.zeros_like(p), torch.zeros_like(p), 0, []
    for _ in range(epochs):
        total = 0.0
        for first in range(0, y.size, batch):
            xb, tb = x[first:first + batch], t[first:first + batch]
            w1, b1, w2, b2, w3, b3 = (p[e - n:e] for e, n in zip(ends, sizes))
            w1, w2 = w1.view(64, 8), w2.view(64, 64)
            h1 = torch.relu(xb @ w1.T + b1)
            h2 = torch.relu(h1 @ w2.T + b2)
            z = h2 @ w3 + b3
            total = total + torch.nn.functional.binary_cross_entropy_with_logits(z, tb, reduction="sum")
            dz = (torch.sigmoid(z) - tb) / tb.numel()
            d2 = dz[:, None] * w3[None, :] * (h2 > 0)
            d1 = (d2 @ w2) * (h1 > 0)
            grad = torch.cat([(d1.T @ xb).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), dz @ h2,
                              dz.sum()[None], torch.zeros(p.numel() - int(ends[-1]), dtype=p.dtype, device=p.device)])
            step += 1
            m = 0.9 * m + 0.1 * grad
            v = 0.999 * v + 0.001 * grad * grad
            p = p - LEARNING_RATE * (m / (1 - 0.9**step)) / (torch.sqrt(v / (1 - 0.999**step)) + 1e-8)
        losses.append(total / y.size)
    return p.cpu().numpy(), torch.stack(losses).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "score":
        s = prepare(case, seed)
        return {"scores": _score_exact(s["programs"], s["features"]), "actions": None}
    if kind == "train":
        s = prepare(case, seed)
        params, losses = _train_exact(s["params"], s["x"], s["y"], case["epochs"], case["batch"], s["seed"])
        return {"params": params, "losses": losses}
    if kind == "pheromone":
        s = prepare(case, seed)
        trails = torch.clamp(s["trails"].double() * RETENTION, min=TAU_MIN)
        parent, primary = s["parent"].long(), s["primary"].long()
        succ, pred = torch.empty_like(parent), torch.empty_like(parent)
        succ[parent], pred[parent] = torch.roll(parent, -1), torch.roll(parent, 1)
        on = (primary == succ[:, None]) | (primary == pred[:, None])
        trails = torch.where(on, torch.clamp(trails + DEPOSIT, max=TAU_MAX), trails)
        return {"trails": trails, "products": trails * s["eta"].double()}
    # tours, lengths and counters are whole numbers that every tree has to
    # reproduce; the prior's rows follow from them
    return None
