"""What users of this framework have it do, as cases to time: MaxCut solves of
one graph, TSP solves, and batched MaxCut, each one complete solve through the
Python binding of the C ABI (sbx.py), from the seeded initial state to the
agents' cuts, tours or spins.

Graphs, agents, time steps and precisions are those of the repository's own
configurations and tests: Erdos-Renyi 800 (FP32), the 100 x 100 torus (BF16
and FP32), R-MAT up to 2^20 vertices, 30-city tours, the batch of 512
instances, weighted graphs, FP64.  The long runs use whole schedules of fewer
SB steps than the 10,000 to 20,000 of those configurations, so that a pass
stays under two seconds; the work per step is the same.
"""
import math
import os
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sparse-ising-solver_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
import sbx  # noqa: E402

# Single MaxCut: graph and its size, weights (unit: +1, pm1: +-1, real),
# agents, state precision, dt, SB steps, and the options of the solve.
MAXCUT = dict(family="maxcut", graph="er", n=800, degree=48.0, weights="unit", agents=1024,
              precision="f32", dt=0.1, steps=1000, fused=1, update_window=0, trace=0, state=0, oneshot=0)
TSP = dict(family="tsp", cities=30, agents=1024, precision="f32", dt=0.1, steps=5000, penalty=1.0)
BATCH = dict(family="batch", kind="mixed", instances=512, nmin=100, nmax=20000, agents=64,
             precision="bf16", dt=0.5, steps=1000)


def listed():
    def mc(name, **kw):
        return dict(MAXCUT, name=name, **kw)

    return [
        # The smallest call: a graph arrives, is solved once with few agents
        # and read back (problem creation, solve, spins): latency counts.
        mc("er200_oneshot_f32", n=200, degree=10.0, weights="pm1", agents=64, steps=300, state=1, oneshot=1),
        # The reference's plain use: default precision, a Gset-sized random
        # graph, 1024 agents, 10,000 steps.
        mc("er800_f32", steps=10000),
        # A lattice spin glass with the early exit, 16-bit state.
        mc("torus100_bf16", graph="torus", n=10000, weights="pm1", precision="bf16", dt=0.5, steps=20000,
           update_window=1),
        # The same lattice in the default precision.
        mc("torus100_f32", graph="torus", n=10000, weights="pm1", dt=0.5, steps=4000),
        # The largest single graph: power-law degrees, heavy and isolated rows.
        mc("rmat20_bf16", graph="rmat", n=1 << 20, agents=256, precision="bf16", dt=0.5, steps=1500),
        # A mid-sized power-law graph with the best cut recorded every window
        # (time-to-target studies).
        mc("rmat16_f16_trace", graph="rmat", n=1 << 16, agents=256, precision="f16", dt=0.5, steps=2000, trace=1),
        # A weighted graph (real edge weights, as .mtx files carry them) with
        # odd sizes: rows and agents that fill no tile.
        mc("rgg2917_real_f32", graph="rgg", n=2917, degree=12.0, weights="real", agents=200, steps=2000, state=1),
        # The FP64 mode, unfused steps: reproducing the reference's numbers.
        mc("er301_f64_unfused", n=301, degree=12.0, weights="pm1", agents=33, precision="f64", steps=500, fused=0,
           state=1),
        # Tours: 30 cities, 1024 agents, 16-bit state and the default FP32.
        dict(TSP, name="tsp30_f16", precision="f16", steps=20000, penalty=1.5),
        dict(TSP, name="tsp29_f32", cities=29, agents=1000),
        # Many graphs of uneven size in one call (the throughput workload),
        # and a smaller batch in the default precision.
        dict(BATCH, name="batch512_bf16", steps=1500),
        dict(BATCH, name="batch96_f32", instances=96, nmax=3000, precision="f32", steps=2000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(work_per_step, most, precision):
    """SB steps (whole windows of 100) that keep a pass within the listed ones."""
    budget = {"f64": 4e10, "f32": 4e11}.get(precision, 8e11)
    return max(100, min(most, int(budget / work_per_step) // 100 * 100))


def draw(rng):
    kind = rng.choice(["er", "rgg", "torus", "rmat", "tsp", "batch"])
    if kind == "tsp":
        prec = rng.choice(["f16", "bf16", "f32"])
        cities, agents = rng.randint(5, 32), _log(rng, 32, 1024)
        return dict(TSP, cities=cities, agents=agents, precision=prec, penalty=rng.choice([1.0, 1.5]),
                    steps=_steps(4.0 * cities ** 3 * 1024, 20000, prec))
    if kind == "batch":
        b = dict(BATCH, kind=rng.choice(["mixed", "mixed", "torus"]), instances=_log(rng, 8, 512),
                 nmax=_log(rng, 1000, 20000), agents=rng.choice([32, 64, 64, 100]),
                 precision=rng.choice(["bf16", "bf16", "f16", "f32"]))
        rows = b["instances"] * (b["nmax"] - b["nmin"]) / math.log(b["nmax"] / b["nmin"])
        return dict(b, steps=_steps(64.0 * rows * 31, 1500, b["precision"]))
    c = dict(MAXCUT, graph=kind, agents=_log(rng, 32, 1024), precision=rng.choice(["f32", "bf16", "f16"]),
             dt=rng.choice([0.1, 0.5]), weights=rng.choice(["unit", "pm1"]))
    if kind == "torus":
        c.update(n=rng.randint(20, 120) ** 2, degree=4.0, weights="pm1", update_window=rng.randint(0, 1))
    elif kind == "rmat":
        c.update(n=1 << rng.randint(12, 20), degree=8.0, weights="unit", agents=_log(rng, 32, 256),
                 trace=rng.randint(0, 1))
    else:
        c.update(n=_log(rng, 100, 10000), degree=float(rng.randint(6, 48)), state=rng.randint(0, 1))
        if kind == "rgg":
            c.update(weights=rng.choice(["pm1", "real"]))
            if c["weights"] == "real":
                c.update(n=_log(rng, 100, 4000), degree=float(rng.randint(6, 24)))
        if c["n"] <= 400 and c["agents"] <= 128 and rng.random() < 0.3:
            c.update(precision="f64", fused=0)
    return dict(c, steps=_steps(c["agents"] * c["n"] * (c["degree"] + 8.0), 10000, c["precision"]))


def _rmat(scale, edge_factor, seed):
    """R-MAT (0.57, 0.19, 0.19), weights +1, self loops and duplicates
    removed, made on the GPU."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    n, m = 1 << scale, edge_factor << scale
    u = torch.zeros(m, dtype=torch.int64, device=dev)
    v = torch.zeros(m, dtype=torch.int64, device=dev)
    for _ in range(scale):
        x = torch.rand(m, generator=g, device=dev)
        q = (x >= 0.57).long() + (x >= 0.76).long() + (x >= 0.95).long()
        u, v = (u << 1) | (q >> 1), (v << 1) | (q & 1)
    keep = u != v
    lo, hi = torch.minimum(u, v)[keep], torch.maximum(u, v)[keep]
    e = torch.unique(lo * n + hi)
    r, c = e // n, e % n
    both = torch.sort(torch.cat([e, c * n + r]))[0]
    deg = torch.bincount(both // n, minlength=n)
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = torch.cumsum(deg, 0).cpu().numpy()
    col = (both % n).to(torch.int32).cpu().numpy()
    return sbx.Graph(n, rowptr, col, np.ones(col.size), float(e.numel()))


def _real_weights(g, seed):
    """Symmetric real weights in [-1, 1], one per edge, from the seed."""
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(g.n, dtype=np.int64), np.diff(g.rowptr))
    key = np.minimum(r, g.col) * g.n + np.maximum(r, g.col)
    edges, at = np.unique(key, return_inverse=True)
    w = rng.uniform(-1.0, 1.0, edges.size)
    return sbx.Graph(g.n, g.rowptr, g.col, w[at], float(w.sum()))


def _graph(case, seed):
    kind, n = case["graph"], case["n"]
    if kind == "rmat":
        return _rmat(n.bit_length() - 1, 4, seed)
    if kind == "torus":
        side = math.isqrt(n)
        return sbx.gen_torus(side, side, seed=seed)
    pm1 = case["weights"] != "unit"
    if kind == "rgg":
        g = sbx.gen_rgg(n, case["degree"], seed=seed)
    else:
        g = sbx.gen_er(n, min(1.0, case["degree"] / (n - 1)), pm1=pm1, seed=seed)
    return _real_weights(g, seed) if case["weights"] == "real" else g


def _batch_graphs(case, seed):
    """n log-uniform in [nmin, nmax]; Erdos-Renyi and geometric graphs in
    turn, average degree uniform in [6, 40] (or tori), weights +-1."""
    rng = np.random.default_rng(seed)
    specs = []
    for i in range(case["instances"]):
        n = int(round(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        specs.append((i, n, float(rng.uniform(6, 40))))

    def make(spec):
        i, n, deg = spec
        if case["kind"] == "torus":
            return sbx.gen_torus(max(3, math.isqrt(n)), max(3, math.isqrt(n)), seed=seed + i)
        if i % 2:
            return sbx.gen_rgg(n, deg, seed=seed + i)
        return sbx.gen_er(n, min(1.0, deg / (n - 1)), pm1=True, seed=seed + i)

    with ThreadPoolExecutor(8) as pool:
        return list(pool.map(make, specs))


def prepare(case, seed):
    ctx = sbx.Context(0)
    st = {"case": case, "ctx": ctx}
    if case["family"] == "tsp":
        xc, yc = sbx.gen_cities(case["cities"], 1000.0, seed=seed)
        st["prob"] = ctx.tsp_problem_cities(xc, yc, sbx.DIST_EUC_2D_FLOAT, A=1.0, penalty_scale=case["penalty"])
        st["prm"] = sbx.params(dt=case["dt"], steps=case["steps"], agents=case["agents"],
                               precision=case["precision"], seed=seed & 0x7fffffff)
    elif case["family"] == "batch":
        graphs = _batch_graphs(case, seed)
        st["probs"] = [ctx.problem(g) for g in graphs]
        st["agents"] = [case["agents"]] * len(graphs)
        st["prm"] = sbx.params(dt=case["dt"], steps=case["steps"], precision=case["precision"],
                               seed=seed & 0x7fffffff)
    else:
        st["graph"] = _graph(case, seed)
        if not case["oneshot"]:
            st["prob"] = ctx.problem(st["graph"])
        st["prm"] = sbx.params(dt=case["dt"], steps=case["steps"], agents=case["agents"], fused=case["fused"],
                               update_window=case["update_window"], trace=case["trace"],
                               precision=case["precision"], seed=seed & 0x7fffffff)
    return st


STATS = ("min", "max", "mean", "std", "ps")


def run(st):
    case, ctx = st["case"], st["ctx"]
    if case["family"] == "batch":
        res, vals, _ = ctx.solve_batch(st["probs"], st["agents"], st["prm"])
        return {"values": vals, "stats": np.array([[r[k] for k in STATS] for r in res])}
    prob = ctx.problem(st["graph"]) if case.get("oneshot") else st["prob"]
    res, vals = ctx.solve(prob, st["prm"])
    if case["family"] == "tsp":
        tours, valid = ctx.tours(case["cities"], case["agents"])
        return {"lengths": vals, "tours": tours, "valid": valid}
    out = {"values": vals, "stats": [res[k] for k in STATS], "steps": res["steps_run"],
           "bifurcated": res["bifurcated"]}
    if case["trace"]:
        steps, best, _ = ctx.trace()
        out["trace"] = [steps, best]
    if case["state"]:
        out["x"], out["y"], out["spins"] = ctx.state(prob.n, case["agents"])
    if case.get("oneshot"):
        prob.close()
    return out


def work(case):
    """Per SB step and agent: one addition per stored entry of J, about eight
    operations per spin (force, clamp, drift, kick); TSP: the distance product
    2 N^3 and the same eight per spin.  Bytes: the matrix once, the results."""
    if case["family"] == "tsp":
        n3 = case["cities"] ** 3
        return {"bytes": 8.0 * case["cities"] ** 2 + 4.0 * case["agents"] * (case["cities"] + 3),
                "flops": case["steps"] * case["agents"] * (2.0 * n3 + 8.0 * case["cities"] ** 2)}
    if case["family"] == "batch":
        rows = case["instances"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        nnz = rows * (4.0 if case["kind"] == "torus" else 23.0)
    else:
        rows, nnz = float(case["n"]), case["n"] * (4.0 if case["graph"] == "torus" else
                                                   7.8 if case["graph"] == "rmat" else case["degree"])
    state = 20.0 * rows * case["agents"] if case.get("state") else 0.0
    return {"bytes": 8.0 * nnz + 4.0 * rows + 8.0 * case["agents"] * case.get("instances", 1) + state,
            "flops": case["steps"] * case["agents"] * (nnz + 8.0 * rows)}


def _glibc_rand(seed, count):
    """The first `count` values of rand() after srand(seed) (TYPE_3)."""
    r = [0] * (344 + count)
    r[0] = seed if seed else 1
    for i in range(1, 31):
        r[i] = (16807 * r[i - 1]) % 2147483647
    for i in range(31, 34):
        r[i] = r[i - 31]
    for i in range(34, 344 + count):
        r[i] = (r[i - 31] + r[i - 3]) & 0xffffffff
    return np.array(r[344:], np.int64) >> 1


def exact(case, seed):
    """The FP64 cases restated in numpy: the SB dynamics with every force
    taken from the signs of the step before, and the exact cut.  The other
    precisions' runs are chaotic over their hundreds to thousands of steps, so
    64 bits says nothing of them."""
    if case["family"] != "maxcut" or case["precision"] != "f64" or case["n"] > 400 or case["trace"] or \
            case["update_window"] or case["steps"] % 100:
        return None
    g, A, dt, steps = _graph(case, seed), case["agents"], case["dt"], case["steps"]
    n = g.n
    J = np.zeros((n, n))
    np.add.at(J, (np.repeat(np.arange(n), np.diff(g.rowptr)), g.col), g.val)
    nn = float(n) * n
    mean = g.val.sum() / nn
    var = (np.square(g.val - mean).sum() + (nn - g.nnz) * mean * mean) / (nn - 1.0)
    c0 = dt * (0.7 / (math.sqrt(var) * math.sqrt(n)))
    v = (_glibc_rand(seed & 0x7fffffff, 2 * n * A) / 2147483647.0 * 2.0 - 1.0) / 10.0
    x, y = v[0::2].reshape(n, A).copy(), v[1::2].reshape(n, A).copy()

    def spins():
        return np.where(np.signbit(x), -1.0, 1.0)

    y += dt * -1.0 * x
    x += dt * y
    for k in range(steps):
        p = 1.025 * k / steps
        if not case["fused"]:
            y += dt * (p - 1) * x
            x += dt * (p + 1) * y
        y += c0 * -(J @ spins())
        out = np.abs(x) > 1.0
        x, y = np.where(out, spins(), x), np.where(out, 0.0, y)
        if case["fused"]:
            p = min(p, 1.0)
            x += dt * (p + 1) * y
            y += dt * (p - 1) * x
    s = spins()
    cut = -0.5 * (0.5 * (s * (J @ s)).sum(axis=0) - g.wsum)
    best = cut.max()
    dev = math.sqrt(np.square(cut - cut.mean()).sum() / (A - 1))
    out = {"values": cut, "stats": [cut.min(), best, cut.mean(), dev, float((cut == best).sum()) / A],
           "steps": None, "bifurcated": None}
    if case["state"]:
        out.update(x=x.reshape(-1), y=y.reshape(-1), spins=None)
    return out
