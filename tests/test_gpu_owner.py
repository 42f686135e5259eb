"""Counting from the later endpoint of each DAG edge (csrc/rows.cu), the default route of
the triangle plan: bitmaps of the out-lists of vertices of degree > 112, merges for the
others.  Sizes sit at the edges of its tiers: degrees around 112, in-neighbour counts
around the 512 of one unit and several units, suffixes around the longest that one thread
tests (12) and the 128 elements of one warp pass.  Counts equal closed forms, the oracle
and the task tiers (forced by a fixed schedule)."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _complete(n):
    iu = np.triu_indices(n, 1)
    return n, iu[0].astype(np.int32), iu[1].astype(np.int32)


def _join(core, leaves, per_leaf):
    """A complete graph on `core` vertices and `leaves` more, each joined to the first
    `per_leaf` core vertices: those have core - 1 + leaves neighbours."""
    n, s, d = _complete(core)
    ls = np.repeat(np.arange(core, core + leaves, dtype=np.int32), per_leaf)
    ld = np.tile(np.arange(per_leaf, dtype=np.int32), leaves)
    return core + leaves, np.concatenate([s, ls]), np.concatenate([d, ld])


@pytest.mark.parametrize("n", [2, 3, 14, 15, 33, 64, 65, 66, 67, 112, 113, 114, 115, 128, 129, 130, 195, 300])
def test_complete_graphs(ctx, n):
    g = ctx.graph_from_edges(*_complete(n))
    assert ctx.count(g, "triangle") == math.comb(n, 3)
    g.close()


@pytest.mark.parametrize("core,leaves,per", [(70, 441, 70), (70, 442, 70), (70, 443, 3),
                                             (20, 1600, 13), (140, 5000, 14), (3, 70000, 2)])
def test_hubs_of_several_units(ctx, core, leaves, per):
    g = ctx.graph_from_edges(*_join(core, leaves, per))
    assert ctx.count(g, "triangle") == math.comb(core, 3) + leaves * math.comb(per, 2)
    g.close()


@pytest.mark.parametrize("gen,args", [("rmat", (9, 4)), ("rmat", (12, 16)), ("er", (3001, 3001 * 40)),
                                      ("er", (500, 60000)), ("ba", (3312, 3)),
                                      ("chung_lu", (20001, 2.1, 3000.0, 20.0))])
def test_oracle_and_task_tiers(xgm, orc, ctx, gen, args):
    nv, src, dst = getattr(xgm, "gen_" + gen)(*args, seed=29)
    rowptr, col = orc.build_csr(nv, src, dst)
    g = ctx.graph_from_edges(nv, src, dst)
    drow, dcol = orc.orient(rowptr, col)
    want = orc.count("tc", drow, dcol)
    got, st = ctx.count(g, "triangle", with_stats=True)
    assert got == want
    assert st["tasks"] == int(np.count_nonzero(np.diff(drow) >= 2))
    assert ctx.count(g, "triangle", policy=xgm.SCHED_FIXED, variant=xgm.VAR_WARP) == want
    g.close()


def test_no_edges_and_batched_ranks(xgm, ctx):
    none = np.zeros(0, dtype=np.int32)
    g = ctx.graph_from_edges(7, none, none)
    assert ctx.count(g, "triangle") == 0
    g.close()


@pytest.mark.parametrize("core,leaves,per", [(66, 0, 0), (70, 441, 70), (70, 443, 3),
                                             (20, 1600, 13), (140, 5000, 14), (3, 70000, 2)])
def test_participation_of_hubs(ctx, core, leaves, per):
    """Diamonds and tailed triangles from triangles per edge, at the same edges of the tiers:
    every pair of the core is an edge of core - 2 triangles inside it, and of `leaves` more
    when both are joined to them."""
    g = ctx.graph_from_edges(*_join(core, leaves, per))
    t_core = [core - 2 + (leaves if j < per else 0) for j in range(core) for _ in range(j)]
    diamonds = sum(math.comb(t, 2) for t in t_core) + leaves * per * math.comb(max(per - 1, 0), 2)
    assert ctx.count(g, "diamond") == diamonds
    # per vertex: triangles x (degree - 2)
    t_in = math.comb(core - 1, 2) + leaves * max(per - 1, 0)
    tailed = per * t_in * (core - 1 + leaves - 2) + (core - per) * math.comb(core - 1, 2) * (core - 3)
    tailed += leaves * math.comb(per, 2) * (per - 2) if per > 2 else 0
    assert ctx.count(g, "tailedtriangle") == tailed
    g.close()


@pytest.mark.parametrize("gen,args", [("rmat", (11, 16)), ("er", (500, 60000)),
                                      ("er", (20001, 160000)),
                                      ("chung_lu", (20001, 2.1, 3000.0, 20.0))])
def test_participation_oracle_and_task_tiers(xgm, orc, ctx, gen, args):
    nv, src, dst = getattr(xgm, "gen_" + gen)(*args, seed=43)
    rowptr, col = orc.build_csr(nv, src, dst)
    g = ctx.graph_from_edges(nv, src, dst)
    for kind, pattern in (("diamond", "diamond"), ("tailed", "tailedtriangle")):
        want = orc.count(kind, rowptr, col)
        assert ctx.count(g, pattern) == want
        assert ctx.count(g, pattern, policy=xgm.SCHED_FIXED, variant=xgm.VAR_WARP) == want
    g.close()


@pytest.mark.parametrize("core", [24, 25, 26, 27])
def test_short_lists_with_hubs(xgm, orc, ctx, core):
    # largest out-degree 23 to 26, around the line below which no edge takes a bitmap unit,
    # with hubs of degree above 112 either side of it
    nv, src, dst = _join(core, 300, core - 4)
    rowptr, col = orc.build_csr(nv, src, dst)
    g = ctx.graph_from_edges(nv, src, dst)
    assert g.info()["max_out_degree"] == core - 1
    assert ctx.count(g, "triangle") == math.comb(core, 3) + 300 * math.comb(core - 4, 2)
    assert ctx.count(g, "4-clique") == math.comb(core, 4) + 300 * math.comb(core - 4, 3)
    assert ctx.count(g, "diamond") == orc.count("diamond", rowptr, col)
    assert xgm.MotifSolver(g, 4) == [int(c) for c in orc.motif(4, rowptr, col)]
    g.close()
