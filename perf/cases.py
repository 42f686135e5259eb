"""Performance cases: what a program that counts patterns with this engine has it do.

Every case goes through the Python mirror of the C ABI (x-gminer_gb300/__init__.py): the
reference-shaped solvers, the counting calls of a context, the batched count, and the
upload of a host graph.  Graphs come from the engine's seeded generators in the families
that the tests and bench.py use (R-MAT, Erdos-Renyi, Chung-Lu, Barabasi-Albert), cleaned
on the GPU; a program holds the built graph, the trained schedule and the plans and then
counts, so those are made in prepare().  One process keeps one context, as the solvers do.

Counts are whole numbers.  work() gives the bytes of the graph that a count reads (the
oriented rows for the clique plans, the whole adjacency otherwise), each once: the path
computes no floating-point operation.
"""
from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

xgm = importlib.import_module("x-gminer_gb300")

# GLUMIN's generated 5-vertex plans and the 5-vertex patterns compiled from their shape
GLUMIN_PLANS = ("P6", "P7", "P8", "P10", "P13", "P15", "P17", "P20", "P22")
COMPILED_PLANS = ("5-house", "5-solid-house", "5-double-triangle")
BATCH_PATTERNS = ["triangle", "4-clique", "diamond"]


def listed():
    return [
        # the smallest call: triangles of a citation-network-sized graph (a few thousand
        # vertices); launches and the read-back are all there is
        {"name": "tc_ba_3312", "op": "tc", "family": "ba", "n": 3312, "deg": 3},
        # a small graph's whole 4-motif census: many short passes one after the other
        {"name": "motif4_er_20011", "op": "motif", "k": 4, "family": "er", "n": 20011, "deg": 16},
        # triangles of a social-network-like graph of a million vertices
        {"name": "tc_rmat20", "op": "tc", "family": "rmat", "scale": 20, "deg": 16},
        # the headline workload: 4-cliques at R-MAT scale 22 under the trained schedule
        {"name": "clique4_rmat22_learned", "op": "clique", "k": 4, "learned": True,
         "family": "rmat", "scale": 22, "deg": 16},
        # deeper cliques through CliqueSolver, plain schedule
        {"name": "clique5_rmat20", "op": "clique", "k": 5, "learned": False,
         "family": "rmat", "scale": 20, "deg": 16},
        {"name": "clique6_rmat16", "op": "clique", "k": 6, "learned": False,
         "family": "rmat", "scale": 16, "deg": 16},
        # edge-induced motifs (ScSolver): a power-law graph of odd size, and the even
        # degrees of an Erdos-Renyi graph
        {"name": "diamond_cl_1500001", "op": "sc", "pattern": "diamond", "family": "cl",
         "n": 1500001, "deg": 32, "dmax": 50000},
        {"name": "cycle4_er_1m", "op": "sc", "pattern": "rectangle", "family": "er",
         "n": 1 << 20, "deg": 32},
        # the 4-motif census of a mid-size skewed graph
        {"name": "motif4_rmat19", "op": "motif", "k": 4, "family": "rmat", "scale": 19, "deg": 16},
        # a 5-vertex plan of GLUMIN's set (5-half-house), vertex-induced
        {"name": "plan_p7_rmat12", "op": "plan", "pattern": "P7", "induced": False,
         "family": "rmat", "scale": 12, "deg": 8},
        # batched counting of thousands of small graphs, three patterns each
        {"name": "batch_ba_4096_learned", "op": "batch", "graphs": 4096, "learned": True},
        # a host graph that is uploaded, counted once and dropped
        {"name": "upload_clique4_rmat20", "op": "upload", "k": 4, "family": "rmat", "scale": 20,
         "deg": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, n_hi, scale_hi, families=("rmat", "er", "cl", "ba")):
    fam = rng.choice(families)
    if fam == "rmat":
        return {"family": "rmat", "scale": rng.randint(10, scale_hi), "deg": rng.randint(5, 16)}
    n = _log_int(rng, 1000, n_hi) | 1
    if fam == "ba":
        return {"family": "ba", "n": min(n, 200001), "deg": rng.randint(3, 8)}
    if fam == "er":
        return {"family": "er", "n": n, "deg": rng.randint(6, 32)}
    return {"family": "cl", "n": n, "deg": rng.randint(8, 32),
            "dmax": max(50, min(50000, n // rng.randint(20, 60)))}


def draw(rng):
    op = rng.choice(["tc", "clique", "clique", "sc", "sc", "motif", "plan", "batch", "upload"])
    if op == "tc":
        return {"op": "tc", **_draw_graph(rng, 1500001, 21)}
    if op == "clique":
        k = rng.choice([4, 4, 4, 5, 5, 6, 7])
        scale = {4: 21, 5: 19, 6: 16, 7: 14}[k]
        # families that hold k-cliques (an Erdos-Renyi graph this sparse has none)
        families = ("rmat", "cl", "ba") if k == 4 else ("rmat", "cl")
        return {"op": "clique", "k": k, "learned": k < 6 and rng.random() < 0.5,
                **_draw_graph(rng, {4: 1500001, 5: 1000001}.get(k, 100001), scale, families)}
    if op == "sc":
        return {"op": "sc", "pattern": rng.choice(["diamond", "rectangle", "tailedtriangle"]),
                **_draw_graph(rng, 1500001, 20)}
    if op == "motif":
        return {"op": "motif", "k": rng.choice([3, 4, 4]), **_draw_graph(rng, 1000001, 19)}
    if op == "plan":
        compiled = rng.random() < 0.3
        g = ({"family": "rmat", "scale": rng.randint(9, 11 if compiled else 12), "deg": 8}
             if rng.random() < 0.5 else
             {"family": "er", "n": _log_int(rng, 1000, 65536) | 1, "deg": rng.randint(8, 16)})
        return {"op": "plan", "pattern": rng.choice(COMPILED_PLANS if compiled else GLUMIN_PLANS),
                "induced": compiled, **g}
    if op == "batch":
        return {"op": "batch", "graphs": _log_int(rng, 16, 4096), "learned": rng.random() < 0.5}
    return {"op": "upload", "k": rng.choice([3, 4]),
            **_draw_graph(rng, 1000001, 20, ("rmat", "cl", "ba"))}


@functools.lru_cache(maxsize=None)
def _context():
    return xgm.Context(0)


@functools.lru_cache(maxsize=None)
def _trained():
    return xgm.trained_schedule(_context())


def _edges(case, seed):
    fam, deg = case["family"], case["deg"]
    if fam == "rmat":
        return xgm.gen_rmat(case["scale"], deg, seed=seed)
    if fam == "er":
        return xgm.gen_er(case["n"], case["n"] * deg // 2, seed=seed)
    if fam == "cl":
        return xgm.gen_chung_lu(case["n"], 2.1, float(case["dmax"]), float(deg), seed=seed)
    return xgm.gen_ba(case["n"], deg, seed=seed)


def prepare(case, seed):
    ctx, op = _context(), case["op"]
    state = {"case": case, "ctx": ctx, "sched": _trained() if case.get("learned") else {}}
    if op == "batch":
        vo, _, src, dst = xgm.gen_ba_batch(case["graphs"], 100, 5000, 3, 8, seed=seed)
        state["batch"] = ctx.batch_from_edges(vo, src, dst)
        state["plans"] = [ctx.plan(p) for p in BATCH_PATTERNS]
        return state
    nv, src, dst = _edges(case, seed)
    g = ctx.graph_from_edges(nv, src, dst)
    if op == "upload":  # the program has the cleaned graph in pinned host memory
        rowptr, col = g.download()
        g.close()
        keep = [torch.from_numpy(a).pin_memory() for a in (rowptr, col)]
        state["pinned"] = keep
        state["rowptr"], state["col"] = (t.numpy() for t in keep)
        state["plan"] = ctx.plan(f"{case['k']}-clique")
        return state
    state["graph"] = g
    if op == "plan":
        state["plan"] = ctx.plan(case["pattern"], induced=case["induced"])
    elif op == "clique":
        state["plan"] = ctx.plan(f"{case['k']}-clique")
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    op = case["op"]
    if op == "batch":
        return ctx.count_batched(state["batch"], state["plans"], **state["sched"])
    if op == "upload":
        g = ctx.graph_from_csr(state["rowptr"], state["col"])
        n = ctx.count(g, state["plan"])
        info = g.info()
        g.close()
        return {"count": n, **info}
    g = state["graph"]
    if op == "tc":
        return xgm.TCSolver(g)
    if op == "clique":
        if case["learned"]:
            return ctx.count(g, state["plan"], **state["sched"])
        return xgm.CliqueSolver(g, case["k"])
    if op == "sc":
        return xgm.ScSolver(g, case["pattern"])
    if op == "motif":
        return xgm.MotifSolver(g, case["k"])
    return ctx.count(g, state["plan"])


def work(case):
    if case["op"] == "batch":
        # log-uniform sizes in [100, 5000], 3 to 8 edges per vertex: about 1,252 vertices
        # and 6,900 edges a graph
        nv, m, out = case["graphs"] * 1252, case["graphs"] * 6900, case["graphs"] * 24
    else:
        nv = (1 << case["scale"]) if case["family"] == "rmat" else case["n"]
        m = nv * case["deg"] // (2 if case["family"] in ("er", "cl") else 1)
        out = 48
    oriented = case["op"] in ("tc", "clique")
    # a 16-byte row descriptor per vertex, 4 bytes per entry
    return {"bytes": 16 * nv + 4 * m * (1 if oriented else 2) + out, "flops": 0}


def exact(case, seed):
    """Triangles of a small graph from its dense adjacency matrix in 64 bits; None where
    that matrix is too large or another pattern is counted."""
    if case["op"] != "tc":
        return None
    nv = (1 << case["scale"]) if case["family"] == "rmat" else case["n"]
    if nv > 4096:
        return None
    nv, src, dst = _edges(case, seed)
    a = np.zeros((nv, nv))
    a[src, dst] = 1.0
    a[dst, src] = 1.0
    np.fill_diagonal(a, 0.0)
    t = torch.from_numpy(a)
    return int(round(float((t @ t).mul_(t).sum()) / 6.0))
