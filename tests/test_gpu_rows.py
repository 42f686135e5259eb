"""Cliques of 4 to 7 vertices from stored rows (csrc/rows.cu), the default route of the
clique plans: rows from the owner kernel, counted as 0/1 matrices in 32 x 32 blocks.  Sizes
sit at its edges: out-degrees around 32 (word / team tasks), 512 (team / wide tasks) and
1,024 (the last stored); rows of around 32 (a matrix in registers), 128 (one warp's), 512
(a team's) and more members; a multiple of 32 and one more.  Counts equal closed forms, the
oracle and the task kernel (forced by a fixed schedule)."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _complete(n):
    iu = np.triu_indices(n, 1)
    return n, iu[0].astype(np.int32), iu[1].astype(np.int32)


@pytest.mark.parametrize("n,kmax", [(4, 7), (7, 7), (17, 7), (18, 7), (32, 7), (33, 7), (34, 7),
                                    (35, 7), (64, 7), (65, 7), (66, 7), (97, 6), (129, 6),
                                    (130, 6), (131, 6), (161, 6), (257, 5), (513, 5), (514, 5),
                                    (515, 5), (545, 5), (1024, 5), (1025, 5)])
def test_complete_graphs(ctx, n, kmax):
    g = ctx.graph_from_edges(*_complete(n))
    for k in range(4, kmax + 1):
        assert ctx.count(g, f"{k}-clique") == math.comb(n, k), k
    g.close()


def test_vertices_above_the_row_capacity(ctx):
    """Out-degrees up to 1,107: 83 vertices above the row store's 1,024 run in the task
    kernel (enough for its hub kernel), the rest from rows."""
    n = 1108
    g = ctx.graph_from_edges(*_complete(n))
    assert ctx.count(g, "4-clique") == math.comb(n, 4)
    g.close()


@pytest.mark.parametrize("gen,args", [("rmat", (9, 8)), ("rmat", (12, 16)), ("er", (400, 30000)),
                                      ("er", (1200, 300000)), ("ba", (5000, 7)),
                                      ("chung_lu", (20001, 2.1, 3000.0, 20.0))])
def test_oracle_and_task_kernel(xgm, orc, ctx, gen, args):
    nv, src, dst = getattr(xgm, "gen_" + gen)(*args, seed=31)
    g = ctx.graph_from_edges(nv, src, dst)
    rowptr, col = orc.build_csr(nv, src, dst)
    drow, dcol = orc.orient(rowptr, col)
    for k in (4, 5, 6):
        got, st = ctx.count(g, f"{k}-clique", with_stats=True)
        assert got == ctx.count(g, f"{k}-clique", policy=xgm.SCHED_FIXED, variant=xgm.VAR_WARP)
        assert st["tasks"] == int(np.count_nonzero(np.diff(drow) >= k - 1))
        if k == 4 or len(dcol) < 120000:
            assert got == orc.count(f"clique{k}", drow, dcol)
    g.close()


def test_buffers_follow_the_graph(xgm, ctx):
    """One context counts a large and then a small graph, and the large one again."""
    graphs = [xgm.gen_rmat(13, 16, seed=3), xgm.gen_ba(300, 4, seed=3)]
    gs = [ctx.graph_from_edges(*x) for x in graphs]
    first = [ctx.count(g, "4-clique") for g in gs]
    assert [ctx.count(g, "4-clique") for g in gs] == first
    assert ctx.count_kernels(gs[0], "4-clique") >= 2
    for g in gs:
        g.close()
