"""Performance cases: the work a user of this package has it do.

Every case is one pass through a public entry point: an exact evaluation of
one graph (from a host array, as the reference's annealing loop calls
``evaluation()``, or of an adjacency already on the device), a batch of graphs
in one launch, some steps of the annealer, or the proposal filter's network.
``listed()`` names the cases, ``draw()`` makes more of the same ranges,
``prepare()`` builds what a program has in hand before the call (seeded graphs
of the shapes the package's generators and benchmark use), ``run()`` is the
call itself, ``work()`` what it cannot do without, and ``exact()`` the answer
in 64 bits by plain torch or numpy.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import graphgolf_b200 as gg
from graphgolf_b200 import graphs
from graphgolf_b200._native import ggb_result, last_error, load


def listed():
    return [
        # The reference's smallest published graphs (256 vertices, degree 4):
        # the latency of one evaluation() call of an annealing loop.
        {"name": "general_n256_d4", "kind": "general", "nodes": 256, "degree": 4, "groups": 1, "centres": 0,
         "entry": "host"},
        # The small annealing configuration: 1024 vertices, degree 8, called
        # once per step by a host annealing loop.
        {"name": "general_n1024_d8", "kind": "general", "nodes": 1024, "degree": 8, "groups": 1, "centres": 0,
         "entry": "host"},
        # The reference's -v 16 -g 15 runs: 15 symmetry groups of 256 vertices
        # and 16 added centres.
        {"name": "centres_n3856_d6", "kind": "general", "nodes": 3856, "degree": 6, "groups": 15, "centres": 16,
         "entry": "host"},
        # The non-regular evaluator at an uneven size and an odd degree.
        {"name": "nonregular_n5002_d7", "kind": "nonregular", "nodes": 5002, "degree": 7, "drop": 400},
        # The grid configuration: 100 x 100 lattice, degree 4, edge length 3;
        # evaluated once per step of a 100 000-step annealing run.
        {"name": "grid_100x100_d4_r3", "kind": "grid", "width": 100, "height": 100, "degree": 4, "length": 3},
        # The headline: one large graph, adjacency resident on the device.
        {"name": "general_n65536_d16", "kind": "general", "nodes": 65536, "degree": 16, "groups": 1, "centres": 0,
         "entry": "device"},
        # Its symmetric variant: 16 groups, 4096 sources, from the host.
        {"name": "symmetric_n65536_d16_g16", "kind": "general", "nodes": 65536, "degree": 16, "groups": 16,
         "centres": 0, "entry": "host"},
        # The largest: four times the headline's vertices, ids past 16 bits.
        {"name": "general_n262144_d12", "kind": "general", "nodes": 262144, "degree": 12, "groups": 1, "centres": 0,
         "entry": "device"},
        # The mixed batch: a 4096-vertex base graph and 256 candidates of 512
        # to 16384 vertices, uploaded and evaluated in one launch.
        {"name": "batch_257_d12", "kind": "batch", "candidates": 256, "degree": 12, "n_lo": 512, "n_hi": 16384},
        # Plain annealing on the device, the small configuration: one candidate
        # per step, Metropolis with cooling.
        {"name": "anneal_plain_n1024_d8", "kind": "anneal", "nodes": 1024, "degree": 8, "candidates": 1,
         "proposals": 1, "compose": 0, "hill": False, "steps": 200},
        # Learned annealing as configured: the top 64 of 4096 proposals are
        # evaluated exactly, every step trains the filter's network.
        {"name": "anneal_learned_n16384_d12", "kind": "anneal", "nodes": 16384, "degree": 12, "candidates": 64,
         "proposals": 4096, "compose": 64, "hill": False, "steps": 8},
        # The filter's network trained on one step's evaluated candidates.
        {"name": "filter_train_64", "kind": "filter", "rows": 64, "steps": 8},
    ]


def _log(rng, lo, hi):
    """An integer, uniform in its logarithm over [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["general", "general", "general", "symmetric", "centres", "nonregular", "grid", "large", "batch",
                       "plain", "batched", "learned", "filter", "rank"])
    if kind == "general":
        n, d = _log(rng, 64, 65536), rng.randint(3, 16)
        return {"kind": "general", "nodes": n + (n * d) % 2, "degree": d, "groups": 1, "centres": 0,
                "entry": rng.choice(["host", "device"])}
    if kind == "symmetric":
        g, d = rng.choice([2, 4, 8, 16]), rng.choice([4, 6, 8, 10, 12, 16])
        return {"kind": "general", "nodes": g * 2 * _log(rng, 32, 2048), "degree": d, "groups": g, "centres": 0,
                "entry": rng.choice(["host", "device"])}
    if kind == "centres":
        g, c = rng.randint(1, 16), 2 * rng.randint(1, 24)
        return {"kind": "general", "nodes": g * 2 * _log(rng, 16, 512) + c, "degree": rng.randint(4, 12), "groups": g,
                "centres": c, "entry": "host"}
    if kind == "nonregular":
        n = 2 * _log(rng, 64, 8192)
        return {"kind": "nonregular", "nodes": n, "degree": rng.randint(5, 14), "drop": n // rng.randint(10, 40)}
    if kind == "grid":
        return {"kind": "grid", "width": 2 * _log(rng, 5, 64), "height": _log(rng, 10, 128),
                "degree": rng.choice([4, 6, 8]), "length": rng.randint(3, 5)}
    if kind == "large":
        return {"kind": "general", "nodes": 2 * _log(rng, 32768, 98304), "degree": rng.randint(7, 14), "groups": 1,
                "centres": 0, "entry": "device"}
    if kind == "batch":
        return {"kind": "batch", "candidates": _log(rng, 8, 256), "degree": rng.randint(4, 16),
                "n_lo": _log(rng, 64, 1024), "n_hi": _log(rng, 2048, 16384)}
    if kind == "plain":
        n = 2 * _log(rng, 128, 8192)
        return {"kind": "anneal", "nodes": n, "degree": rng.randint(4, 12), "candidates": 1, "proposals": 1,
                "compose": 0, "hill": rng.random() < 0.5, "steps": rng.randint(20, 100)}
    if kind in ("batched", "learned"):
        k = 16 * rng.randint(2, 16)
        return {"kind": "anneal", "nodes": 2 * _log(rng, 512, 8192), "degree": rng.randint(8, 14), "candidates": k,
                "proposals": k if kind == "batched" else 16 * rng.randint(32, 256), "compose": k,
                "hill": rng.random() < 0.5, "steps": rng.randint(2, 8)}
    return {"kind": "filter", "rows": 16 * rng.randint(1, 16 if kind == "filter" else 256),
            "steps": rng.randint(1, 16) if kind == "filter" else 0}


# ---- inputs -----------------------------------------------------------------


def _graph(case, seed):
    n, d = case["nodes"], case["degree"]
    if case["groups"] > 1 and not case["centres"]:
        return graphs.symmetric_regular(n, d, case["groups"], seed)
    return graphs.random_regular(n, d, seed)


def _filter_data(rows, seed):
    """Features and labels like the annealer's: 32 values of order one, labels
    of a few units around zero."""
    r = np.random.default_rng(seed)
    x = r.uniform(-1.0, 1.0, (rows, 32)).astype(np.float32)
    t = (2.0 * x[:, 0] - x[:, 5] + x[:, 7] * x[:, 11] + r.normal(0.0, 0.5, rows)).astype(np.float32)
    return x, t


def prepare(case, seed):
    seed = int(seed) % (1 << 31) + 1
    kind = case["kind"]
    if kind == "general":
        g = _graph(case, seed)
        s = {"kind": kind, "case": case, "adj": g.adj, "based": (case["nodes"] - case["centres"]) // case["groups"]}
        if case["entry"] == "device":
            s["dev"] = torch.from_numpy(g.adj).cuda()
        return s
    if kind == "nonregular":
        g = graphs.random_regular(case["nodes"], case["degree"], seed)
        _, adj, deg = graphs.nonregular(g, case["drop"], seed)
        return {"kind": kind, "adj": adj, "deg": deg}
    if kind == "grid":
        g = graphs.grid_regular(case["width"], case["height"], case["degree"], case["length"], seed)
        return {"kind": kind, "adj": g.adj, "rh": g.rotate_hash}
    if kind == "batch":
        w = graphs.batch_workload(case["candidates"], case["degree"], case["n_lo"], case["n_hi"],
                                  base_nodes=2 * (case["n_hi"] // 8), seed=seed)
        return {"kind": kind, "adjs": [g.adj for g in w], "batch": gg.Batch([g.nodes for g in w], case["degree"])}
    if kind == "anneal":
        g = graphs.random_regular(case["nodes"], case["degree"], seed)
        a = gg.Annealer(g, candidates=case["candidates"], proposals=case["proposals"], compose=case["compose"],
                        seed=seed)
        if not case["hill"]:
            a.schedule(temp=100.0, cooling=0.9995, hill_climbing=False)
        return {"kind": kind, "annealer": a, "steps": case["steps"],
                "learned": case["proposals"] > case["candidates"]}
    rows = case["rows"]
    x, t = _filter_data(rows, seed)
    return {"kind": kind, "net": gg.FilterNet(rows, seed), "x": x, "t": t, "steps": case["steps"]}


# ---- one pass ---------------------------------------------------------------


def _answer(r):
    return {"connected": bool(r.connected), "diameter": int(r.diameter), "total": int(r.total), "aspl": float(r.aspl)}


def run(state):
    kind = state["kind"]
    if kind == "general":
        c = state["case"]
        if c["entry"] == "host":
            return _answer(gg.evaluate(state["adj"], state["based"], c["groups"], c["centres"]))
        r = ggb_result()
        rc = load().ggb_eval_general_device(c["nodes"], state["based"], c["groups"], c["degree"],
                                            state["dev"].data_ptr(), c["centres"], None, ctypes.byref(r))
        if rc != 0:
            raise gg.EvaluationError(rc, last_error())
        return _answer(r)
    if kind == "nonregular":
        return _answer(gg.evaluate_nonregular(state["adj"], state["deg"]))
    if kind == "grid":
        return _answer(gg.evaluate_grid(state["adj"], state["rh"]))
    if kind == "batch":
        res = state["batch"].evaluate(state["adjs"])
        return {"connected": np.array([r.connected for r in res]), "diameter": np.array([r.diameter for r in res]),
                "total": np.array([r.total for r in res]), "aspl": np.array([r.aspl for r in res])}
    if kind == "anneal":
        a = state["annealer"]
        st = a.run(state["steps"])
        out = {"step": st.step, "accepts": st.accepts, "moved_swaps": st.moved_swaps, "evals": st.evals,
               "unevaluated": st.unevaluated, "cur_diam": st.cur_diam, "best_diam": st.best_diam,
               "cur_total": st.cur_total, "best_total": st.best_total, "temp": st.temp, "edges": a.edges()}
        if state["learned"]:
            out["predicted"], out["label"] = a.last_step()
        return out
    net = state["net"]
    if state["steps"] == 0:
        return {"y": net.forward(state["x"])}
    loss = net.train(state["x"], state["t"], state["steps"])
    return {"loss": np.float32(loss), "params": net.params}


# ---- what a pass cannot do without ------------------------------------------


def _sizes(case):
    """(vertices, sources, degree) of the evaluations of one pass."""
    kind = case["kind"]
    if kind == "general":
        return [(case["nodes"], (case["nodes"] - case["centres"]) // case["groups"], case["degree"])]
    if kind == "nonregular":
        return [(case["nodes"], case["nodes"], case["degree"])]
    if kind == "grid":
        n = case["width"] * case["height"]
        return [(n, n, case["degree"])]
    # a batch: the mean of N and N^2 for N log-uniform over the range
    lo, hi = float(case["n_lo"]), float(case["n_hi"])
    k = math.log(hi / lo)
    n, n2 = (hi - lo) / k, (hi * hi - lo * lo) / (2.0 * k)
    return [(n, n2 / n, case["degree"])] * (case["candidates"] + 1)


def work(case):
    """bytes: each input read once, each output written once.  flops: for an
    evaluation, one decision per (vertex, source) pair; for the network, the
    multiply-adds of its layers (forward, and twice that backward)."""
    kind = case["kind"]
    if kind == "filter":
        per_row = 2 * (32 * 256 + 256 * 256 + 256)
        if case["steps"] == 0:
            return {"bytes": case["rows"] * (32 + 1) * 4 + (32 * 256 + 256 * 256) * 2, "flops": case["rows"] * per_row}
        params = 32 * 256 + 256 + 256 * 256 + 256 + 256 + 1
        return {"bytes": case["steps"] * (case["rows"] * 33 * 4 + 6 * params * 4),
                "flops": case["steps"] * 3 * case["rows"] * per_row}
    if kind == "anneal":
        n, d, s = case["nodes"], case["degree"], case["steps"]
        # a step reads the graph and decides the distances of one graph; the
        # candidates evaluated against it change few of them
        return {"bytes": s * n * d * 4 + 2 * n * d * 4, "flops": s * n * n}
    return {"bytes": sum(n * d * 4 for n, _, d in _sizes(case)), "flops": sum(n * src for n, src, _ in _sizes(case))}


# ---- the answer in 64 bits --------------------------------------------------


def _popcount(x):
    """Set bits of every int64 word."""
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    x = x + (x >> 8)
    x = x + (x >> 16)
    return (x + (x >> 32)) & 0x7F


def _distances(adj, sources, split):
    """Sums of the distances from every source to the vertices below `split`
    and to the others, and the largest distance: breadth-first search of 4096
    sources at a time on bit sets."""
    n = adj.shape[0]
    at = torch.from_numpy(np.ascontiguousarray(adj, dtype=np.int64)).cuda()
    lo = hi = diam = 0
    for s0 in range(0, len(sources), 4096):
        src = torch.tensor(sources[s0:s0 + 4096], dtype=torch.int64, device="cuda")
        m, words = len(src), (len(src) + 63) // 64
        row = torch.zeros((n, words), dtype=torch.int64, device="cuda")
        i = torch.arange(m, device="cuda")
        row[src, i // 64] = torch.ones_like(i) << (i % 64)
        last, level = -1, 0
        while True:
            per = _popcount(row).sum(1)
            reached = int(per.sum())
            if reached == n * m:
                break
            if reached == last:
                return None
            last = reached
            lo += split * m - int(per[:split].sum())
            hi += (n - split) * m - int(per[split:].sum())
            new = row.clone()
            for j in range(at.shape[1]):
                new |= row[at[:, j]]
            row = new
            level += 1
        diam = max(diam, level)
    return lo, hi, diam


def _exact_graph(adj, based=None, groups=1, centres=0):
    n = adj.shape[0]
    based = n if based is None else based
    split = based * groups
    got = _distances(adj, list(range(based)), split)
    if got is None:
        return None
    lo, hi, diam = got
    total = groups * (lo + 2 * hi)
    if centres:
        _, among, d2 = _distances(adj, list(range(n - centres, n)), split)
        total, diam = total + among, max(diam, d2)
    return {"connected": True, "diameter": diam, "total": total, "aspl": total / ((n - 1) * n)}


def _network64(p, x):
    w1, b1, w2, b2, w3, b3 = (p[a:b] for a, b in ((0, 8192), (8192, 8448), (8448, 73984), (73984, 74240),
                                                  (74240, 74496), (74496, 74497)))
    h1 = np.maximum(x @ w1.reshape(256, 32).T + b1, 0.0)
    z2 = h1 @ w2.reshape(256, 256).T + b2
    h2 = np.maximum(z2, 0.0)
    return h2 @ w3 + b3[0], h1, z2, h2, w2.reshape(256, 256), w3


def _exact_filter(case, seed):
    seed = int(seed) % (1 << 31) + 1
    x32, t32 = _filter_data(case["rows"], seed)
    x, t = x32.astype(np.float64), t32.astype(np.float64)
    p = gg.FilterNet(case["rows"], seed).params.astype(np.float64)
    if case["steps"] == 0:
        return {"y": _network64(p, x)[0]}
    m1, m2, loss = np.zeros_like(p), np.zeros_like(p), 0.0
    for k in range(1, case["steps"] + 1):
        y, h1, z2, h2, w2, w3 = _network64(p, x)
        loss = float(np.mean((y - t) ** 2))
        dy = 2.0 * (y - t) / len(t)
        dz2 = (z2 > 0) * dy[:, None] * w3[None, :]
        dz1 = (dz2 @ w2) * (h1 > 0)
        g = np.concatenate([(dz1.T @ x).ravel(), dz1.sum(0), (dz2.T @ h1).ravel(), dz2.sum(0), h2.T @ dy, [dy.sum()]])
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        p = p - 1e-3 * (m1 / (1 - 0.9 ** k)) / (np.sqrt(m2 / (1 - 0.999 ** k)) + 1e-8)
    return {"loss": loss, "params": p}


def exact(case, seed):
    kind = case["kind"]
    if kind == "filter":
        return _exact_filter(case, seed)
    if kind == "anneal":   # whole numbers, and a search whose course has no closed form
        return None
    if kind == "batch":
        seed = int(seed) % (1 << 31) + 1
        w = graphs.batch_workload(case["candidates"], case["degree"], case["n_lo"], case["n_hi"],
                                  base_nodes=2 * (case["n_hi"] // 8), seed=seed)
        got = [_exact_graph(g.adj) for g in w]
        if any(r is None for r in got):
            return None
        return {k: np.array([r[k] for r in got]) for k in got[0]}
    s = prepare(case, seed)
    if kind == "general":
        return _exact_graph(s["adj"], s["based"], case["groups"], case["centres"])
    return _exact_graph(s["adj"])
