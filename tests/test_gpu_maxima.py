"""Large point sets through the GPU-wide maxima pass (pmdd_b200/csrc/engine/maxima.cuh):
oversized destinations with int32 and int64 objectives."""
from __future__ import annotations

import numpy as np
import pytest

import pmdd_b200 as P
from pmdd_b200 import instances

pytestmark = pytest.mark.gpu


def _knapsack_text(profits, weights, cap):
    rows = [f"{profits.shape[1]} 1 {profits.shape[0]}"] + [" ".join(map(str, r)) for r in profits]
    return "\n".join(rows + [" ".join(map(str, weights)) + f" {cap}"]) + "\n"


@pytest.mark.parametrize("nobjs,n", [(4, 40), (5, 30), (6, 28), (7, 25), (8, 24)])
def test_oversized_destinations_int64_match_int32(nobjs, n):
    """Profits times 2,000,000 need 64-bit sums; the frontier scales with them."""
    profits, weights, cap = instances.knapsack_arrays(n, nobjs, 77 + nobjs)
    st = {}
    small = P.enumerate_dd(P.DecisionDiagram.from_text(_knapsack_text(profits, weights, cap), 1, nobjs), stats=st)
    assert st["work_tile_candidates_total"] < st["work_candidates_total"]  # some destinations left the tiles
    wide = P.enumerate_dd(
        P.DecisionDiagram.from_text(_knapsack_text(profits * 2_000_000, weights, cap), 1, nobjs))
    assert small.dtype == np.int32 and wide.dtype == np.int64
    want = small.astype(np.int64) * 2_000_000
    assert np.array_equal(wide[np.lexsort(wide.T[::-1])], want[np.lexsort(want.T[::-1])])
