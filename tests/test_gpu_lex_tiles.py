"""The three-objective tile kernel (lex_items.cuh) where its chunks can go wrong: small
objective ranges (equal values of objective 1 and equal points inside a chunk and across
chunks), antichains in objectives 1 and 2 (full staircases), and int64 points."""
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


@pytest.mark.parametrize("method", [1, 3])
@pytest.mark.parametrize("hi", [2, 4, 12, 1000])
@pytest.mark.parametrize("n", [14, 27, 40])
def test_ties_and_duplicates(n, hi, method):
    rng = np.random.default_rng(100 * n + hi)
    profits = rng.integers(0, hi, size=(3, n))
    weights = rng.integers(1, 60, size=n)
    dd = P.DecisionDiagram.from_text(_text(profits, weights, int(weights.sum()) // 2), 1, 3)
    got = P.enumerate_dd(dd, method=method)
    assert np.array_equal(oracle.sorted_set(got), oracle.sorted_set(oracle.enumerate(dd, method)))
    assert len(np.unique(got, axis=0)) == len(got)


@pytest.mark.parametrize("antichain", [False, True])
@pytest.mark.parametrize("n", [16, 30, 44])
def test_int64_points_match_int32(n, antichain):
    """Profits times 1,500,000 need 64-bit sums; the frontier scales with them."""
    profits, weights, cap = instances.knapsack_arrays(n, 3, 500 + n)
    if antichain:
        n = min(n, 22)
        profits, weights = profits[:, :n], weights[:n]
        profits[2] = 1001 - profits[1]
        cap = int(weights.sum()) // 2
    small = P.enumerate_dd(P.DecisionDiagram.from_text(_text(profits, weights, cap), 1, 3))
    scaled = profits.astype(np.int64) * 1_500_000
    wide = P.enumerate_dd(P.DecisionDiagram.from_text(_text(scaled, weights, cap), 1, 3))
    assert small.dtype == np.int32 and wide.dtype == np.int64
    want = small.astype(np.int64) * 1_500_000
    assert np.array_equal(wide[np.lexsort(wide.T[::-1])], want[np.lexsort(want.T[::-1])])
