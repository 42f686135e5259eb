"""4-cycles of vertices whose wedges are few for the ids they are spread over (csrc/cycle4.cu:
hash passes over ranges of ids instead of tiles of counters), and of heavy vertices in batches,
whose graphs begin at other ids.  Against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RIMS = 1 << 20


def _wheel(seed, hubs, spokes):
    """Two million-odd ids: RIMS rim vertices with two spokes each; `spokes` lists (number,
    rims each) of two kinds, hubs (kind, spokes taken).  A hub's wedges end at its spokes' rims,
    all over the ids."""
    rng = np.random.default_rng(seed)
    src, dst, nv, kinds = [], [], RIMS, []
    for n, each in spokes:
        ids = np.arange(nv, nv + n)
        nv += n
        kinds.append(ids)
        src.append(np.repeat(ids, each))
        dst.append(rng.integers(0, RIMS, n * each))
    for kind, take in hubs:
        src.append(np.full(take, nv))
        dst.append(rng.choice(kinds[kind], take, replace=False))
        nv += 1
    # every rim in some rows, so that ranks of rims spread over all ids
    src.append(np.arange(RIMS))
    dst.append(rng.permutation(RIMS))
    return nv, np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)


@pytest.mark.parametrize("seed,hubs,spokes", [
    # (a) up to 64 and to 512 lower neighbours: about 20,000 and 30,000 wedges, and past the line
    (1, [(0, 20), (0, 30), (0, 31), (0, 64), (1, 500), (1, 512)], [(1200, 1000), (3000, 40)]),
    # (b) 513 to 2,048 lower neighbours: in passes, in one pass, past the line
    (2, [(1, 513), (1, 600), (1, 800), (1, 2048), (0, 600)], [(700, 900), (3000, 40)]),
    # (c) above: units of a hub and a tile
    (3, [(1, 2049), (1, 2600), (1, 2900), (0, 520)], [(600, 500), (3000, 30)]),
    # (d) rows of unequal spread: few spokes with many rims among many with few
    (4, [(0, 9), (1, 2000), (1, 1000), (1, 515)], [(10, 9000), (2500, 12)])])
def test_spread_out_wedges(xgm, orc, ctx, seed, hubs, spokes):
    nv, src, dst = _wheel(seed, hubs, spokes)
    rowptr, col = orc.build_csr(nv, src, dst)
    want = orc.count("cycle4", rowptr, col)
    g = ctx.graph_from_edges(nv, src, dst)
    assert ctx.count(g, "rectangle") == want
    g.close()


def test_even_graph(xgm, orc, ctx):
    nv, src, dst = xgm.gen_er(1 << 20, 90 << 19, seed=6)  # about 8,100 wedges at the top ranks
    rowptr, col = orc.build_csr(nv, src, dst)
    g = ctx.graph_from_edges(nv, src, dst)
    assert ctx.count(g, "rectangle") == orc.count("cycle4", rowptr, col)
    g.close()


def test_batches_of_heavy_vertices(xgm, orc, ctx):
    rng = np.random.default_rng(7)
    parts, off = [], [0]

    def add(n, s, d):
        parts.append((np.asarray(s, np.int32), np.asarray(d, np.int32), n))
        off.append(off[-1] + n)

    for i in range(60):  # ids before and between the heavy graphs
        add(*xgm.gen_ba(2000 + i, 4, seed=i))
        if i % 6 == 0:
            n = [300, 700, 1500, 3000, 5200][(i // 6) % 5]  # hub degrees below and above 2,048
            hubs = [np.full(n - 1, 0), np.full(n // 2, 1), np.full(n // 3, 2)]
            ends = [np.arange(1, n), rng.choice(np.arange(3, n), n // 2, replace=False),
                    rng.choice(np.arange(3, n), n // 3, replace=False)]
            _, s, d = xgm.gen_er(n, 12 * n, seed=i + 1)
            add(n, np.concatenate(hubs + [s]), np.concatenate(ends + [d]))
    b = ctx.batch_from_edges(np.array(off, np.int64),
                             np.concatenate([p[0] + o for p, o in zip(parts, off)]).astype(np.int32),
                             np.concatenate([p[1] + o for p, o in zip(parts, off)]).astype(np.int32))
    got = ctx.count_batched(b, ["rectangle"])[:, 0].tolist()
    want = [orc.count("cycle4", *orc.build_csr(n, s, d)) for s, d, n in parts]
    assert got == want
    b.close()


@pytest.mark.parametrize("spokes", [8192, 8193, 9001, 20000])
def test_one_id_in_more_rows_than_a_table_takes(xgm, orc, ctx, spokes):
    """Two hubs with the same spokes: one v2 has as many wedges as there are spokes, the others
    one each, all over the ids."""
    rng = np.random.default_rng(9)
    sp = np.arange(RIMS, RIMS + spokes)
    c, v0 = RIMS + spokes, RIMS + spokes + 1
    parts = [(np.full(spokes, c), sp), (np.full(spokes, v0), sp),
             (np.full(10, v0), rng.choice(RIMS, 10, replace=False)),
             (sp, rng.integers(0, RIMS, spokes)), (np.arange(RIMS), rng.permutation(RIMS))]
    nv = RIMS + spokes + 2
    src = np.concatenate([p[0] for p in parts]).astype(np.int32)
    dst = np.concatenate([p[1] for p in parts]).astype(np.int32)
    want = orc.count("cycle4", *orc.build_csr(nv, src, dst))
    assert want >= spokes * (spokes - 1) // 2
    g = ctx.graph_from_edges(nv, src, dst)
    assert ctx.count(g, "rectangle") == want
    g.close()
