"""The autotuner's table is never slower than leaving the schedule alone: where the engine's own
choice is the fastest, the table says so and runs it."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_engine_choice_of_a_batch(xgm, ctx):
    vo, _, s, d = xgm.gen_ba_batch(512, 100, 5000, 3, 8, seed=5)
    b = ctx.batch_from_edges(vo, s, d)
    pats = ["triangle", "4-clique", "diamond"]
    base = ctx.count_batched(b, pats)
    res = ctx.autotune(b, pats, reps=2)
    assert res["best_ms"] <= res["heuristic_ms"]
    assert res["variants"] == [xgm.TUNE_ENGINE] * xgm.TUNE_BUCKETS
    got, st = ctx.count_batched(b, pats, policy=xgm.SCHED_TUNED, table=res["table"], with_stats=True)
    assert np.array_equal(got, base) and sum(st["variant_tasks"]) == 0
    b.close()


@pytest.mark.parametrize("pattern", ["triangle", "4-clique", "diamond"])
def test_engine_choice_of_a_graph(xgm, ctx, pattern):
    nv, s, d = xgm.gen_rmat(15, 16, seed=3)
    g = ctx.graph_from_edges(nv, s, d)
    res = ctx.autotune(g, pattern, reps=2)
    assert res["best_ms"] <= res["heuristic_ms"]
    assert res["variants"] == [xgm.TUNE_ENGINE] * xgm.TUNE_BUCKETS
    n, st = ctx.count(g, pattern, policy=xgm.SCHED_TUNED, table=res["table"], with_stats=True)
    assert n == ctx.count(g, pattern) and sum(st["variant_tasks"]) == 0
    assert ctx.motif_count(g, 4) == xgm.MotifSolver(g, 4)
    g.close()


def test_tables_of_variants_run_as_they_are(xgm, ctx):
    nv, s, d = xgm.gen_rmat(12, 16, seed=3)
    g = ctx.graph_from_edges(nv, s, d)
    t = xgm.TuneTable()
    for i in range(xgm.TUNE_BUCKETS):
        t.variant[i] = xgm.VAR_CTA
    want = ctx.count(g, "4-clique")
    n, st = ctx.count(g, "4-clique", policy=xgm.SCHED_TUNED, table=t, with_stats=True)
    assert n == want and st["variant_tasks"][xgm.VAR_CTA] > 0
    t.variant[3] = xgm.TUNE_ENGINE  # an entry among variants is no choice of the engine's
    n, st = ctx.count(g, "4-clique", policy=xgm.SCHED_TUNED, table=t, with_stats=True)
    assert n == want and sum(st["variant_tasks"]) > 0
    g.close()
