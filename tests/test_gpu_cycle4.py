"""Edge-induced 4-cycles (csrc/cycle4.cu) at the edges of its tiers: tasks of up to 64 lower
neighbours and 1,344 wedges (a warp's hash table), 512 lower neighbours and 8,192 wedges (a
CTA's), 2,048 lower neighbours (tiles of counters with cursors), hubs (a unit per tile) and
hubs above 65,535 lower neighbours (32-bit counters).  Counts equal closed forms and the
oracle."""
from __future__ import annotations

from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bipartite(m, n):
    """K_{m,n}: C(m, 2) C(n, 2) 4-cycles; m < n, so the m side ranks highest."""
    s = np.repeat(np.arange(m, dtype=np.int32), n)
    d = np.tile(np.arange(m, m + n, dtype=np.int32), m)
    return m + n, s, d


@pytest.mark.parametrize("m,n", [(2, 2), (2, 3), (2, 64), (2, 65), (3, 64), (21, 64), (22, 64),
                                 (23, 64), (2, 512), (2, 513), (16, 512), (17, 512), (18, 513),
                                 (2, 2048), (2, 2049), (3, 2050), (2, 65535), (2, 65536),
                                 (3, 65537), (2, 50000), (300, 400)])
def test_complete_bipartite(ctx, m, n):
    g = ctx.graph_from_edges(*_bipartite(m, n))
    assert ctx.count(g, "rectangle") == comb(m, 2) * comb(n, 2)
    g.close()


@pytest.mark.parametrize("n", [3, 4, 5, 33, 66, 130, 600])
def test_complete_graphs(ctx, n):
    iu = np.triu_indices(n, 1)
    g = ctx.graph_from_edges(n, iu[0].astype(np.int32), iu[1].astype(np.int32))
    assert ctx.count(g, "rectangle") == 3 * comb(n, 4)
    g.close()


@pytest.mark.parametrize("gen,args", [("rmat", (10, 8)), ("rmat", (14, 16)), ("er", (5001, 160000)),
                                      ("er", (60001, 480000)), ("ba", (20001, 5)),
                                      ("chung_lu", (150001, 2.1, 9000.0, 20.0))])
def test_oracle(xgm, orc, ctx, gen, args):
    nv, src, dst = getattr(xgm, "gen_" + gen)(*args, seed=37)
    rowptr, col = orc.build_csr(nv, src, dst)
    g = ctx.graph_from_edges(nv, src, dst)
    want = orc.count("cycle4", rowptr, col)
    assert ctx.count(g, "rectangle") == want
    assert ctx.count(g, "rectangle") == want  # the counters are left clean
    g.close()
