"""Batched counts on the routes that the batch tests' default sets do not take: the task kernel
without a participation plan, and graphs above the row capacity."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _complete_batch(ctx, sizes):
    off, s, d = [0], [], []
    for n in sizes:
        iu = np.triu_indices(n, 1)
        s.append(iu[0] + off[-1])
        d.append(iu[1] + off[-1])
        off.append(off[-1] + n)
    return ctx.batch_from_edges(np.array(off, np.int64), np.concatenate(s).astype(np.int32),
                                np.concatenate(d).astype(np.int32))


def _want(sizes, k):
    return [math.comb(n, k) for n in sizes]


@pytest.mark.parametrize("kw", [{"group_max": 8}, {"bucket_max": 32}, {"hash_only": True}])
def test_repeated_counts_without_participation(ctx, kw):
    """The task kernel's participation buffers are the batch's, not the captured graph's: a
    replay, another plan set and a plan that needs them follow."""
    sizes = [3, 9, 40, 150]
    b = _complete_batch(ctx, sizes)
    for pat, k in (("triangle", 3), ("4-clique", 4), ("triangle", 3)):
        for _ in range(3):
            assert ctx.count_batched(b, [pat], **kw)[:, 0].tolist() == _want(sizes, k)
    dia = [math.comb(n, 2) * math.comb(n - 2, 2) for n in sizes]
    assert ctx.count_batched(b, ["diamond"], **kw)[:, 0].tolist() == dia
    assert ctx.count_batched(b, ["triangle"], **kw)[:, 0].tolist() == _want(sizes, 3)
    b.close()


def test_default_schedule_above_the_row_capacity(ctx):
    """K(n, n) with the path and one triangle among the second side: each vertex of the first
    has n > 1,024 out-neighbours, one triangle with each of their n edges, one 4-clique."""
    n, small = 1100, 33
    a, c = np.divmod(np.arange(n * n, dtype=np.int64), n)
    path = np.arange(n, 2 * n - 1, dtype=np.int64)
    iu = np.triu_indices(small, 1)
    src = np.concatenate([a, path, [n], iu[0] + 2 * n]).astype(np.int32)
    dst = np.concatenate([n + c, path + 1, [n + 2], iu[1] + 2 * n]).astype(np.int32)
    b = ctx.batch_from_edges(np.array([0, 2 * n, 2 * n + small], np.int64), src, dst)
    want = {"triangle": [n * n + 1, math.comb(small, 3)], "4-clique": [n, math.comb(small, 4)]}
    for pat in want:
        for _ in range(2):
            assert ctx.count_batched(b, [pat])[:, 0].tolist() == want[pat]
    got = ctx.count_batched(b, ["triangle", "4-clique"], use_graph=False)
    assert got[:, 0].tolist() == want["triangle"] and got[:, 1].tolist() == want["4-clique"]
    b.close()
