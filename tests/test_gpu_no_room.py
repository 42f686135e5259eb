"""Counts where there is no room for the row store (the library's test hook says from how many
words on): they run on the task kernel, in the memory that it needs."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import oracle_counts

pytestmark = pytest.mark.gpu

PATTERNS = ["triangle", "4-clique", "diamond", "tailedtriangle", "5-clique", "rectangle"]
KIND = {"triangle": "tc", "4-clique": "clique4", "diamond": "diamond",
        "tailedtriangle": "tailed", "5-clique": "clique5", "rectangle": "cycle4"}


@pytest.fixture
def fresh(xgm):
    c = xgm.Context(0)  # without a store of an earlier call
    yield c
    c.close()


def test_batches(xgm, orc, fresh, monkeypatch):
    vo, eo, s, d = xgm.gen_ba_batch(12, 100, 900, 3, 8, seed=9)
    want = []
    for g in range(len(vo) - 1):
        rowptr, col = orc.build_csr(int(vo[g + 1] - vo[g]), s[eo[g]:eo[g + 1]] - vo[g],
                                    d[eo[g]:eo[g + 1]] - vo[g])
        c = oracle_counts(orc, rowptr, col)
        want.append([c[KIND[p]] for p in PATTERNS])
    want = np.array(want, dtype=np.uint64)
    monkeypatch.setenv("XGM_ROW_STORE_CAP", "100")
    b = fresh.batch_from_edges(vo, s, d)
    model = xgm.Model(fresh, seed=1)
    for _ in range(2):
        got, st = fresh.count_batched(b, PATTERNS, with_stats=True)
        assert np.array_equal(got, want)
        assert sum(st["variant_tasks"]) > 0  # the task kernel ran
    for sub in (["4-clique"], ["triangle"], ["5-clique", "diamond"]):
        cols = [PATTERNS.index(p) for p in sub]
        assert np.array_equal(fresh.count_batched(b, sub), want[:, cols]), sub
    assert np.array_equal(fresh.count_batched(b, PATTERNS, policy=xgm.SCHED_LEARNED, model=model), want)
    # room again: the row kernels, beside the graphs captured before
    monkeypatch.delenv("XGM_ROW_STORE_CAP")
    for _ in range(2):
        got, st = fresh.count_batched(b, PATTERNS, with_stats=True)
        assert np.array_equal(got, want) and sum(st["variant_tasks"]) == 0
    b.close()


def test_graphs(xgm, orc, fresh, monkeypatch):
    nv, src, dst = xgm.gen_rmat(11, 16, seed=4)
    rowptr, col = orc.build_csr(nv, src, dst)
    want = oracle_counts(orc, rowptr, col)
    motifs = [int(c) for c in orc.motif(4, rowptr, col)]
    g = fresh.graph_from_edges(nv, src, dst)
    monkeypatch.setenv("XGM_ROW_STORE_CAP", "100")
    for pat in PATTERNS:
        n, st = fresh.count(g, pat, with_stats=True)
        assert n == want[KIND[pat]], pat
        if pat in ("4-clique", "5-clique"):
            assert sum(st["variant_tasks"]) > 0
    assert fresh.motif_count(g, 4) == motifs
    monkeypatch.delenv("XGM_ROW_STORE_CAP")
    n, st = fresh.count(g, "4-clique", with_stats=True)
    assert n == want["clique4"] and sum(st["variant_tasks"]) == 0
    assert fresh.motif_count(g, 4) == motifs
    g.close()
