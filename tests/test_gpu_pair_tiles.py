"""The pairwise tile kernel (pair_items.cuh): equal and repeated points, where the keep rule
behind its four-at-a-time sweep decides, for every objective count it serves."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pmdd_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hi", [2, 4, 1000])
@pytest.mark.parametrize("nobjs,n", [(1, 24), (2, 31), (4, 26), (5, 22), (6, 20), (7, 17), (8, 17)])
def test_ties_and_duplicates(nobjs, n, hi):
    rng = np.random.default_rng(1000 * nobjs + hi)
    profits = rng.integers(0, hi, size=(nobjs, n))
    weights = rng.integers(1, 50, size=n)
    rows = [f"{n} 1 {nobjs}"] + [" ".join(map(str, r)) for r in profits]
    text = "\n".join(rows + [" ".join(map(str, weights)) + f" {int(weights.sum()) // 2}"]) + "\n"
    dd = P.DecisionDiagram.from_text(text, 1, nobjs)
    got = P.enumerate_dd(dd)
    assert np.array_equal(oracle.sorted_set(got), oracle.sorted_set(oracle.enumerate(dd, 1)))
    assert len(np.unique(got, axis=0)) == len(got)
