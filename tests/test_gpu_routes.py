"""Which kernels an open schedule takes (csrc/count.cu): the owner and row kernels, or the task
kernel on even graphs of long lists.  Counts agree on both sides of each line, the statistics say
which side it was (tasks per variant are the task kernel's), and the owner kernel's own limits
are met: more vertices of degree above 112 than its bitmap has bits, degrees above 262,144."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gen(xgm, name, *args):
    if name == "rings":  # ring lattice: k neighbours either side
        n, k = args
        i = np.repeat(np.arange(n, dtype=np.int64), k)
        return n, i.astype(np.int32), ((i + np.tile(np.arange(1, k + 1), n)) % n).astype(np.int32)
    if name == "cliques":
        c, m = args
        iu = np.triu_indices(m, 1)
        b = np.arange(c, dtype=np.int64)[:, None] * m
        return c * m, (iu[0] + b).ravel().astype(np.int32), (iu[1] + b).ravel().astype(np.int32)
    return getattr(xgm, "gen_" + name)(*args, seed=17)


PATTERNS = ["triangle", "4-clique", "5-clique", "6-clique", "7-clique", "diamond", "tailedtriangle"]


@pytest.mark.parametrize("gen,args,tasks", [
    # (the patterns that the task kernel counts)
    ("er", (1 << 15, 48 << 15), {"4-clique", "5-clique", "6-clique", "7-clique", "diamond",
                                 "tailedtriangle"}),
    ("er", (1 << 16, 24 << 16), {"5-clique", "6-clique", "7-clique"}),
    ("er", (1 << 17, 12 << 17), set()),
    ("er", (150001, 70 * 150001), {"4-clique", "5-clique", "6-clique", "7-clique", "diamond",
                                   "tailedtriangle"}),
    ("rmat", (13, 16), set()),
    ("chung_lu", (100001, 2.1, 2000.0, 32.0), set()),
    ("rings", (1 << 16, 24), set()),
    ("rings", (1 << 16, 33), {"7-clique"}),
    ("cliques", (2000, 60), {"7-clique"}),
])
def test_either_side_of_the_lines(xgm, ctx, gen, args, tasks):
    nv, src, dst = _gen(xgm, gen, *args)
    g = ctx.graph_from_edges(nv, src, dst)
    for pat in PATTERNS:
        if pat == "7-clique" and gen in ("rings", "cliques") and args[0] > 1 << 12 and not tasks:
            continue
        n, st = ctx.count(g, pat, with_stats=True)
        assert (sum(st["variant_tasks"]) > 0) == (pat in tasks), pat
        if gen == "cliques" and pat[0].isdigit():
            assert n == args[0] * math.comb(args[1], int(pat[0]))
        if pat not in ("6-clique", "7-clique"):
            assert n == ctx.count(g, pat, policy=xgm.SCHED_FIXED, variant=xgm.VAR_WARP), pat
    k4 = ctx.count(g, "4-clique")
    census = xgm.MotifSolver(g, 4)
    assert census[5] == k4
    assert census[4] == ctx.count(g, "diamond") - 6 * k4
    g.close()


def test_triangles_of_an_even_graph(xgm, ctx):
    nv, src, dst = xgm.gen_er(1 << 19, 125 << 19, seed=2)  # degree 250: more than the bitmap's
    g = ctx.graph_from_edges(nv, src, dst)
    n, st = ctx.count(g, "triangle", with_stats=True)
    assert sum(st["variant_tasks"]) > 0
    # the owner kernel's count, from another census: 3 x triangles per vertex of the wedges
    wedges, tri = xgm.MotifSolver(g, 3)
    assert tri == n and ctx.count(g, "wedge") == wedges + 3 * tri
    assert n == ctx.count(g, "triangle", policy=xgm.SCHED_FIXED, variant=xgm.VAR_CTA)
    g.close()


def test_more_big_vertices_than_bits(xgm, ctx):
    # 162,000 vertices of degree above 112: those below the top 2^17 (2^18 with credits) are
    # joined a lane an edge
    nv, src, dst = xgm.gen_ba(500001, 64, seed=4)
    g = ctx.graph_from_edges(nv, src, dst)
    for pat in ("triangle", "4-clique", "diamond"):
        n, st = ctx.count(g, pat, with_stats=True)
        assert sum(st["variant_tasks"]) == 0, pat
        assert n == ctx.count(g, pat, policy=xgm.SCHED_FIXED, variant=xgm.VAR_WARP), pat
    g.close()


def test_degrees_above_a_unit_per_level(xgm, ctx):
    # in-neighbours of one vertex in units of 1,024: a unit's second pass keeps the bitmap and
    # the ranks of its first
    core, leaves, per = 30, 300001, 14
    iu = np.triu_indices(core, 1)
    ls = np.repeat(np.arange(core, core + leaves, dtype=np.int32), per)
    ld = np.tile(np.arange(per, dtype=np.int32), leaves)
    g = ctx.graph_from_edges(core + leaves, np.concatenate([iu[0].astype(np.int32), ls]),
                             np.concatenate([iu[1].astype(np.int32), ld]))
    assert g.info()["max_degree"] > 1 << 18
    k4 = math.comb(core, 4) + leaves * math.comb(per, 3)
    t_core = [core - 2 + (leaves if j < per else 0) for j in range(core) for _ in range(j)]
    dia = sum(math.comb(t, 2) for t in t_core) + leaves * per * math.comb(per - 1, 2)
    assert ctx.count(g, "triangle") == math.comb(core, 3) + leaves * math.comb(per, 2)
    assert ctx.count(g, "4-clique") == k4
    assert ctx.count(g, "5-clique") == math.comb(core, 5) + leaves * math.comb(per, 4)
    assert ctx.count(g, "diamond") == dia
    census = xgm.MotifSolver(g, 4)
    assert census[5] == k4 and census[4] == dia - 6 * k4
    g.close()


def test_no_edges(xgm, ctx):
    none = np.zeros(0, dtype=np.int32)
    g = ctx.graph_from_edges(7, none, none)
    for pat in PATTERNS + ["rectangle", "wedge", "P7", "P10"]:
        assert ctx.count(g, pat) == 0, pat
    assert xgm.MotifSolver(g, 3) == [0, 0] and xgm.MotifSolver(g, 4) == [0] * 6
    g.close()
    b = ctx.batch_from_edges(np.array([0, 3, 9], np.int64), none, none)
    pats = ["triangle", "4-clique", "diamond", "5-clique", "rectangle"]
    got, st = ctx.count_batched(b, pats, with_stats=True)
    assert not got.any()
    # the owner and row kernels' few launches
    assert st["launches"] < ctx.count_batched(b, pats, group_max=8, with_stats=True)[1]["launches"]
    b.close()


BATCH = ["triangle", "4-clique", "diamond", "tailedtriangle", "5-clique"]


def _batch(ctx, parts):
    off = np.concatenate([[0], np.cumsum([p[0] for p in parts])]).astype(np.int64)
    return ctx.batch_from_edges(off, np.concatenate([p[1] + o for p, o in zip(parts, off)]).astype(np.int32),
                                np.concatenate([p[2] + o for p, o in zip(parts, off)]).astype(np.int32))


@pytest.mark.parametrize("kind,tasks", [("hubs", False), ("rmat", True)])
def test_batches_of_both_routes(xgm, ctx, kind, tasks):
    none = np.zeros(0, np.int32)
    if kind == "hubs":  # hubs of degree above 112, out-degrees above 24, graphs without an edge
        core = [(70, 441, 7), (20, 1600, 13), (140, 500, 14)]
        parts = []
        for c, leaves, per in core:
            iu = np.triu_indices(c, 1)
            parts.append((c + leaves, np.concatenate([iu[0], np.repeat(np.arange(c, c + leaves), per)]),
                          np.concatenate([iu[1], np.tile(np.arange(per), leaves)])))
            parts.append((5, none, none))
        parts += [xgm.gen_ba(1500, 5, seed=i) for i in range(40)]
    else:
        parts = [xgm.gen_rmat(12, 16, seed=i) for i in range(4)] + [(9, none, none)]
    b = _batch(ctx, parts)
    want = []
    for n, s, d in parts:
        g = ctx.graph_from_edges(n, np.asarray(s, np.int32), np.asarray(d, np.int32))
        want.append([ctx.count(g, p, policy=xgm.SCHED_FIXED, variant=xgm.VAR_WARP) for p in BATCH])
        g.close()
    want = np.array(want, np.uint64)
    for sub in (BATCH, ["triangle", "diamond"], ["4-clique"], ["5-clique"], ["tailedtriangle"]):
        cols = [BATCH.index(p) for p in sub]
        for _ in range(2):
            got, st = ctx.count_batched(b, sub, with_stats=True)
            assert np.array_equal(got, want[:, cols]), sub
        if sub != ["5-clique"]:
            assert (sum(st["variant_tasks"]) > 0) == tasks, sub
    b.close()


@pytest.mark.parametrize("core,leaves,per", [(30, 300001, 14), (40, 1000, 33), (3, 9, 2)])
def test_tailed_triangles_of_hubs(xgm, ctx, core, leaves, per):
    """The first has edges in 300,000 triangles between vertices of degree 300,000 (a term above
    32 bits), the second 34 out-neighbours a vertex on average (a warp a vertex), the third 2."""
    iu = np.triu_indices(core, 1)
    ls = np.repeat(np.arange(core, core + leaves, dtype=np.int32), per)
    ld = np.tile(np.arange(per, dtype=np.int32), leaves)
    g = ctx.graph_from_edges(core + leaves, np.concatenate([iu[0].astype(np.int32), ls]),
                             np.concatenate([iu[1].astype(np.int32), ld]))
    t_in = math.comb(core - 1, 2) + leaves * (per - 1)  # triangles of a joined core vertex
    want = per * t_in * (core - 1 + leaves - 2) + (core - per) * math.comb(core - 1, 2) * (core - 3)
    want += leaves * math.comb(per, 2) * max(per - 2, 0)
    n, st = ctx.count(g, "tailedtriangle", with_stats=True)
    assert n == want and sum(st["variant_tasks"]) == 0
    assert ctx.count(g, "tailedtriangle", policy=xgm.SCHED_FIXED, variant=xgm.VAR_WARP) == want
    g.close()
