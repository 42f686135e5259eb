"""Bitmap form of set-operation programs (setbits.cu) at the edges of its kernels.

A hub of each degree at which the form's kernel, word count, row stride or unit split
changes, with sparse neighbourhoods otherwise, against the oracle's plans; and the matching
orders that compiled programs take for the bitmap form against brute force.
"""
from __future__ import annotations

import pytest

from test_gpu_setprog import _hub_graph
from test_setprog import _adj, _random_graph

pytestmark = pytest.mark.gpu

# stream plans (v2 outside N(v0)): P7, P8, P15; bounded and unbounded counts otherwise
QUICK = (6, 7, 8, 9, 13, 14, 17, 19, 20, 22)


@pytest.mark.parametrize("deg", [31, 32, 33, 63, 65, 127, 128, 129, 160, 257, 383, 384, 385, 513,
                                 1023, 1024, 1025])
def test_bitmap_degrees(xgm, ctx, orc, deg):
    rowptr, col = _hub_graph(deg + 1, min(0.3, 6.0 / deg), deg)
    g = ctx.graph_from_csr(rowptr, col)
    plans = QUICK + ((15,) if deg <= 400 else ()) + ((10,) if deg <= 129 else ())
    for pid in plans:
        assert ctx.count(g, f"P{pid}") == orc.glumin5(pid, rowptr, col), pid
    g.close()


@pytest.mark.parametrize("nv,p", [(40, 0.5), (150, 0.6), (260, 0.3)])
def test_dense_graphs(xgm, ctx, orc, nv, p):
    # every vertex in the bitmap form, rows half full: full hash buckets, long v3 lists
    rowptr, col = _random_graph(nv, p, nv)
    g = ctx.graph_from_csr(rowptr, col)
    for pid in (7, 8, 10, 15, 17) if nv < 200 else (8, 17):
        assert ctx.count(g, f"P{pid}") == orc.glumin5(pid, rowptr, col), pid
    g.close()


@pytest.mark.parametrize("nv,deg", [(1200, 13), (1200, 21), (1500, 24), (900, 40), (3000, 100)])
def test_sparse_graphs(xgm, ctx, orc, nv, deg):
    # few steps share a v2: the tables of two-hop vertices are filled to the limit and past
    # it (a pass that does not fit is halved); at degree 24 some vertices have over 32
    rowptr, col = _random_graph(nv, deg / nv, nv + deg)
    g = ctx.graph_from_csr(rowptr, col)
    for pid in (7, 8, 11, 12, 15, 16) if deg < 50 else (7, 8, 12):
        assert ctx.count(g, f"P{pid}") == orc.glumin5(pid, rowptr, col), pid
    g.close()


@pytest.mark.parametrize("edges", [
    [(0, 1), (0, 2), (1, 2), (1, 3), (0, 4)],                  # bull
    [(0, 1), (1, 2), (1, 3), (2, 3), (0, 4)],
    [(0, 1), (0, 2), (1, 2), (1, 3), (2, 3), (0, 4)],
    [(0, 1), (1, 2), (0, 3), (2, 3), (0, 4), (1, 4)],          # house
    [(0, 2), (1, 2), (0, 3), (1, 3), (2, 3), (0, 4), (1, 4)],
])
def test_orders_chosen_for_the_bitmap_form(xgm, ctx, orc, edges):
    a = _adj(edges)
    plan = ctx.plan(a, induced=True, program=True)
    rowptr, col = _random_graph(30, 0.3, 8)
    g = ctx.graph_from_csr(rowptr, col)
    assert ctx.count(g, plan) == orc.occurrences(a, True, rowptr, col)
    g.close()
    rowptr, col = _hub_graph(200, 0.03, 4)
    g = ctx.graph_from_csr(rowptr, col)
    assert ctx.count(g, plan) == orc.program(plan.program, rowptr, col)
    g.close()
