"""Matching orders of compiled programs: which take another order for its bitmap form."""
from __future__ import annotations

import numpy as np
import pytest

N0, N1 = 16, 17  # operands N(v0), N(v1)


def _program(xgm, edges):
    k = max(max(e) for e in edges) + 1
    a = np.zeros((k, k), np.uint8)
    for u, v in edges:
        a[u, v] = a[v, u] = 1
    w = xgm.plan(a, induced=True, program=True).program
    ops = [tuple(int(x) for x in w[12 + 6 * i:18 + 6 * i]) for i in range(int(w[5:9].sum()))]
    return w, ops


def test_four_cycle_keeps_the_shorter_lists(xgm):
    # v2 from N(v0) \ N(v1): a stream of N(v1) would be its bitmap form
    w, ops = _program(xgm, [(0, 1), (0, 2), (1, 3), (2, 3)])
    out, kind, a, b = ops[0][:4]
    assert (kind, a, b) == (1, N0, N1) and int(w[9]) == out


@pytest.mark.parametrize("edges", [
    [(0, 1), (0, 2), (1, 3)],                          # 4-path
    [(0, 1), (0, 2), (0, 3), (1, 4), (2, 4)],          # 5-tailed-square
    [(0, 1), (0, 2), (0, 3), (1, 2), (1, 4), (3, 4)]])  # 5-house
def test_streams_of_the_bitmap_form(xgm, edges):
    w, ops = _program(xgm, edges)
    stream = [o for o in ops if o[1:4] == (1, N1, N0)]
    assert len(stream) == 1 and int(w[9]) == stream[0][0]
