"""The cutset join (couple.cu): value ranges that repeat, int64 points, and a join whose
survivors overflow the running frontier's buffer, so that rounds resume."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pmdd_b200 as P
from pmdd_b200 import instances

pytestmark = pytest.mark.gpu


def _text(profits, weights, cap):
    rows = [f"{profits.shape[1]} 1 {profits.shape[0]}"] + [" ".join(map(str, r)) for r in profits]
    return "\n".join(rows + [" ".join(map(str, weights)) + f" {cap}"]) + "\n"


@pytest.mark.parametrize("hi", [2, 5, 1000])
@pytest.mark.parametrize("nobjs,n", [(1, 20), (2, 30), (3, 30), (4, 24), (5, 20), (6, 18), (7, 16), (8, 16)])
def test_join_matches_the_oracle_and_scales_to_int64(nobjs, n, hi):
    rng = np.random.default_rng(10 * nobjs + hi)
    profits = rng.integers(0, hi, size=(nobjs, n))
    weights = rng.integers(1, 100, size=n)
    cap = int(weights.sum()) // 2
    dd = P.DecisionDiagram.from_text(_text(profits, weights, cap), 1, nobjs)
    got = P.enumerate_dd(dd, method=3)
    assert np.array_equal(oracle.sorted_set(got), oracle.sorted_set(oracle.enumerate(dd, 3)))
    scale = (2**31 - 2) // max(1, hi - 1)
    wide = P.enumerate_dd(P.DecisionDiagram.from_text(_text(profits * scale, weights, cap), 1, nobjs), method=3)
    want = got.astype(np.int64) * scale
    assert wide.dtype == np.int64
    assert np.array_equal(wide[np.lexsort(wide.T[::-1])], want[np.lexsort(want.T[::-1])])


def test_join_that_overflows_its_buffer_matches_top_down():
    dd = P.DecisionDiagram.from_text(instances.knapsack_text(60, 4, 4000), 1, 4)
    assert np.array_equal(oracle.sorted_set(P.enumerate_dd(dd, method=3)),
                          oracle.sorted_set(P.enumerate_dd(dd, method=1)))
