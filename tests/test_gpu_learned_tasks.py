"""The learned schedule's classification through counts: a model whose predictions are known, so
that the tasks per variant are too.  (Counts that the owner and row kernels take need no tasks; a
hub limit, an even graph or roots above the row capacity do.)"""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = 5  # features before the variant one-hot


def _favouring(xgm, ctx, variant, gain=5.0):
    """A model that predicts 12 for every variant but `variant`, and 12 - gain for that one."""
    h, f = xgm.MODEL_HIDDEN, xgm.MODEL_FEATURES
    p = np.zeros(xgm.MODEL_PARAMS, np.float32)
    p[SHAPE + variant] = 1.0       # W1[0][one-hot of the variant]
    p[h * f + h] = -gain           # w2[0], after W1 and b1
    p[h * f + 2 * h] = 12.0        # b2
    m = xgm.Model(ctx, seed=1)
    m.set_params(p)
    return m


def _out_degrees(orc, nv, src, dst):
    rowptr, col = orc.build_csr(nv, src, dst)
    return np.diff(orc.orient(rowptr, col)[0])


def _want(xgm, out, kmin, variant, cap):
    """Tasks per variant: `variant` up to its capacity, by capacity above."""
    w = [0] * xgm.NUM_VARIANTS
    tiers = [(xgm.VAR_WARP, 32), (xgm.VAR_WIDE, 128), (xgm.VAR_CTA, 1024)]
    lo = kmin
    w[variant] += int(np.count_nonzero((out >= lo) & (out <= cap)))
    lo = max(lo, cap + 1)
    for v, c in tiers:
        if c >= lo:
            w[v] += int(np.count_nonzero((out >= lo) & (out <= c)))
            lo = c + 1
    return w


@pytest.mark.parametrize("variant,cap", [("VAR_GROUP", 8), ("VAR_SEARCH", 32), ("VAR_BUCKET", 32),
                                         ("VAR_WARP", 32), ("VAR_CTA", 1024)])
@pytest.mark.parametrize("order", [0, 1])
def test_tasks_per_variant(xgm, orc, ctx, variant, cap, order):
    v = getattr(xgm, variant)
    nv, src, dst = xgm.gen_rmat(12, 16, seed=6)
    out = _out_degrees(orc, nv, src, dst)
    g = ctx.graph_from_edges(nv, src, dst)
    m = _favouring(xgm, ctx, v)
    for pat, k in (("triangle", 3), ("4-clique", 4), ("5-clique", 5)):
        n, st = ctx.count(g, pat, policy=xgm.SCHED_LEARNED, model=m, hub_max=-1, order_by_cost=order,
                          with_stats=True)
        assert n == ctx.count(g, pat)
        assert list(st["variant_tasks"]) == _want(xgm, out, k - 1, v, cap), pat
        # a margin above the predicted gain: the heuristic's variants stay
        n, st = ctx.count(g, pat, policy=xgm.SCHED_LEARNED, model=m, hub_max=-1, order_by_cost=order,
                          margin=6.0, with_stats=True)
        assert list(st["variant_tasks"]) == _want(xgm, out, k - 1, xgm.VAR_WARP, 32), pat
    g.close()


def test_even_graph_under_the_model(xgm, orc, ctx):
    nv, src, dst = xgm.gen_er(1 << 15, 48 << 15, seed=6)
    out = _out_degrees(orc, nv, src, dst)
    g = ctx.graph_from_edges(nv, src, dst)
    m = _favouring(xgm, ctx, xgm.VAR_CTA)
    n, st = ctx.count(g, "4-clique", policy=xgm.SCHED_LEARNED, model=m, with_stats=True)
    assert n == ctx.count(g, "4-clique")
    assert list(st["variant_tasks"]) == _want(xgm, out, 3, xgm.VAR_CTA, 1024)
    g.close()


def test_batches_under_the_model(xgm, ctx):
    vo, _, s, d = xgm.gen_ba_batch(32, 100, 2000, 3, 8, seed=8)
    b = ctx.batch_from_edges(vo, s, d)
    pats = ["triangle", "4-clique", "diamond", "5-clique"]
    want = ctx.count_batched(b, pats)
    m = _favouring(xgm, ctx, xgm.VAR_GROUP)
    for order in (0, 1):
        got, st = ctx.count_batched(b, pats, policy=xgm.SCHED_LEARNED, model=m, hub_max=-1,
                                    order_by_cost=order, with_stats=True)
        assert np.array_equal(got, want)
        assert st["variant_tasks"][xgm.VAR_GROUP] > 0 and st["variant_tasks"][xgm.VAR_CTA] == 0
    b.close()


@pytest.mark.parametrize("order", [0, 1])
def test_roots_above_the_row_capacity(xgm, ctx, order):
    # complete 8-partite graph of parts of 180: out-degrees up to 1,260, beside the row kernels
    r, p = 8, 180
    iu = np.triu_indices(r * p, 1)
    keep = (iu[0] // p) != (iu[1] // p)
    g = ctx.graph_from_edges(r * p, iu[0][keep].astype(np.int32), iu[1][keep].astype(np.int32))
    m = xgm.Model(ctx, seed=3)
    for k, pat in ((4, "4-clique"), (5, "5-clique"), (4, "4-clique")):
        kw = {"policy": xgm.SCHED_LEARNED, "model": m, "order_by_cost": order}
        assert ctx.count_kernels(g, pat, **kw) > 0
        try:
            got = ctx.count(g, pat, **kw)
        except xgm.XgmError as e:  # split hubs of 5-cliques may pass the capacity, as by default
            assert pat == "5-clique" and e.status == xgm.ERR_DEVICE
            with pytest.raises(xgm.XgmError):
                ctx.count(g, pat)
            continue
        assert got == math.comb(r, k) * p ** k == ctx.count(g, pat)
    g.close()


def test_order_of_the_roots_above_the_row_capacity(xgm, ctx):
    # the ordered lists are built by other kernels than the lists in vertex order
    r, p = 8, 180
    iu = np.triu_indices(r * p, 1)
    keep = (iu[0] // p) != (iu[1] // p)
    g = ctx.graph_from_edges(r * p, iu[0][keep].astype(np.int32), iu[1][keep].astype(np.int32))
    m = xgm.Model(ctx, seed=3)
    kernels = [ctx.count_kernels(g, "4-clique", policy=xgm.SCHED_LEARNED, model=m, order_by_cost=o)
               for o in (0, 1)]
    assert kernels[0] == ctx.count_kernels(g, "4-clique")
    assert kernels[1] != kernels[0]
    g.close()


def test_the_trainer_times_the_model(xgm, ctx):
    """Validation and evaluation of a trained model are counts on the kernel that it schedules."""
    import importlib

    tr = importlib.import_module("x-gminer_gb300.train_costmodel")
    nv, src, dst = xgm.gen_rmat(13, 16, seed=6)
    g = ctx.graph_from_edges(nv, src, dst)
    m = _favouring(xgm, ctx, xgm.VAR_CTA)
    for pat in tr.PATTERNS + ["triangle"]:
        n, ms, tasks = tr.timed_count(ctx, g, pat, 1)
        assert n == ctx.count(g, pat) and ms > 0 and sum(tasks) > 0, pat
        _, _, by_model = tr.timed_count(ctx, g, pat, 1, policy=xgm.SCHED_LEARNED, model=m, margin=0.2)
        assert sum(by_model) == sum(tasks) and by_model[xgm.VAR_CTA] == sum(by_model), pat
    g.close()


def test_trained_model_gains_on_the_task_kernel(xgm, ctx):
    """As test_gpu_learned.py's gain on a held-out graph (R-MAT scale 21, seed 77; 3 % for the
    noise of the clock), on the kernel that the model schedules."""
    learned = xgm.trained_schedule(ctx)
    if not learned:
        pytest.skip("costmodel.json absent")
    nv, s, d = xgm.gen_rmat(21, 16, seed=77)
    g = ctx.graph_from_edges(nv, s, d)

    def best(kw):
        ctx.count(g, "4-clique", hub_max=1536, **kw)
        ms = []
        for _ in range(5):
            cnt, st = ctx.count(g, "4-clique", hub_max=1536, with_stats=True, **kw)
            assert sum(st["variant_tasks"]) > 0
            ms.append(st["kernel_ms"] + st["prep_ms"])
        return cnt, min(ms)

    c_h, t_h = best({})
    c_l, t_l = best(learned)
    assert c_l == c_h
    assert t_l <= 1.03 * t_h, f"learned {t_l:.2f} ms vs plain heuristic {t_h:.2f} ms"
    g.close()
