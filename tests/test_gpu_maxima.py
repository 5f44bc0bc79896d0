"""Large point sets through the GPU-wide maxima pass (pmdd_b200/csrc/engine/maxima.cuh):
oversized destinations with int32 and int64 objectives, and standalone sets at the pass's
edges (its smallest set, the sample's size, partial groups) in value ranges that fill the
type or repeat."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
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


@pytest.mark.parametrize("nobjs", range(1, 9))
@pytest.mark.parametrize("n", [320, 321, 327, 1025, 4096, 4097, 9001])
def test_standalone_sets_match_the_keep_rule(nobjs, n):
    rng = np.random.default_rng(1000 * nobjs + n)
    lo, hi = np.iinfo(np.int32).min, np.iinfo(np.int32).max
    front = rng.integers(0, 30_000, size=(n, nobjs))
    front[:, 0] = 40_000 - front[:, 1:].sum(axis=1) // max(1, nobjs - 1)  # many maxima
    sets = {"front": front, "repeated": rng.integers(0, 4, size=(n, nobjs)), "equal": np.full((n, nobjs), lo),
            "full range": rng.integers(lo, hi, size=(n, nobjs), endpoint=True),
            "extremes": rng.choice([lo, -1, 0, hi], size=(n, nobjs))}
    for name, pts in sets.items():
        pts = np.ascontiguousarray(pts, dtype=np.int32)
        got = P.pareto_filter(pts)
        want = pts[oracle.nd_keep(pts)]
        assert np.array_equal(oracle.sorted_set(got), oracle.sorted_set(want)), name
