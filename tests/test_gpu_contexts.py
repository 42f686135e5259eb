"""Contexts are independent, one host thread each (include/xgm.h), also where they count the
same graph: the indexes that a graph builds on first use (row store offsets, plan units and
rows, bucket index, task features) are shared by all of them."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# calls that each build another index of the graph on first use
CALLS = [("4-clique", {}), ("P7", {}), ("6-clique", {}), ("P10", {}),
         ("4-clique", {"bucket_max": 32}), ("motif4", {}), ("5-clique", {"learned": True})]


def _run(c, g, call, model):
    pat, kw = call
    if pat == "motif4":
        return c.motif_count(g, 4)
    if kw.get("learned"):  # a hub limit: the task kernel under the model's schedule
        return c.count(g, pat, policy=1, model=model, hub_max=-1)
    return c.count(g, pat, **kw)


def _all(ctxs, f):
    """f(i, ctxs[i]) on a thread each, all started at once; the exceptions."""
    start, errors = threading.Barrier(len(ctxs)), []

    def body(i):
        try:
            start.wait()
            f(i, ctxs[i])
        except Exception as e:  # noqa: BLE001 - reported by the test
            errors.append(repr(e))

    ts = [threading.Thread(target=body, args=(i,)) for i in range(len(ctxs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return errors


@pytest.fixture(scope="module")
def contexts(xgm):
    cs = [xgm.Context(0) for _ in range(3)]
    yield cs
    for c in cs:
        c.close()


@pytest.mark.parametrize("gen,args", [("rmat", (12, 8)), ("er", (30001, 300000)), ("ba", (3312, 3))])
def test_first_use_of_one_graph_by_several_contexts(xgm, contexts, gen, args):
    nv, src, dst = getattr(xgm, "gen_" + gen)(*args, seed=3)
    models = [xgm.Model(c, seed=2) for c in contexts]
    g0 = contexts[0].graph_from_edges(nv, src, dst)
    want = [_run(contexts[0], g0, call, models[0]) for call in CALLS]
    g0.close()
    for first in range(len(CALLS)):
        # a fresh graph; every thread makes the calls in the same order, from another one each
        # time, so that all meet the same missing index
        g = contexts[first % 3].graph_from_edges(nv, src, dst)
        got = [[None] * len(CALLS) for _ in contexts]

        def work(i, c):
            for k in range(len(CALLS)):
                j = (first + k) % len(CALLS)
                got[i][j] = _run(c, g, CALLS[j], models[i])

        assert _all(contexts, work) == []
        assert got == [want] * len(contexts)
        g.close()


def test_kernel_count_before_the_first_learned_count(xgm, contexts):
    # the kernels of a call are counted by capturing it: the features must be there before
    nv, src, dst = xgm.gen_rmat(12, 8, seed=5)
    c = contexts[0]
    m = xgm.Model(c, seed=2)
    g = c.graph_from_edges(nv, src, dst)
    want = c.count(g, "triangle")
    assert c.count_kernels(g, "triangle", policy=xgm.SCHED_LEARNED, model=m) > 0
    assert c.count(g, "triangle", policy=xgm.SCHED_LEARNED, model=m, hub_max=-1) == want
    g.close()
    assert np.uint64(want) > 0


def _hub(n, leaves):
    """A complete graph on n vertices, the first of which has `leaves` neighbours more."""
    iu = np.triu_indices(n, 1)
    l = np.arange(n, n + leaves, dtype=np.int32)
    return (n + leaves, np.concatenate([iu[0].astype(np.int32), np.zeros(leaves, np.int32)]),
            np.concatenate([iu[1].astype(np.int32), l]))


def test_plans_on_graphs_of_other_degrees_at_once(xgm, contexts):
    """A bitmap-form kernel's shared memory follows the graph's largest degree, and the warp
    kernel's the program: calls of other sizes at the same time must not limit one another."""
    graphs = [_hub(12, 20), _hub(12, 180), _hub(12, 300), _hub(12, 900)]
    jobs = []  # per context: its own graphs and plans
    for c in contexts:
        gs = [c.graph_from_edges(*x) for x in graphs]
        ps = [c.plan(p) for p in ("P7", "P10", "P6", "P15")]
        jobs.append((gs, ps, [[c.count(g, p) for p in ps] for g in gs]))

    def work(i, c):
        gs, ps, want = jobs[i]
        rng = np.random.default_rng(i)
        for a, b in zip(rng.integers(0, len(gs), 1500), rng.integers(0, len(ps), 1500)):
            assert c.count(gs[a], ps[b]) == want[a][b]

    assert _all(contexts, work) == []
    assert jobs[0][2] == jobs[1][2] == jobs[2][2]
    for gs, _, _ in jobs:
        for g in gs:
            g.close()
