"""State dominance where nodes hold many labels: a warp reads its partners' labels 32 at a
time, so frontiers well past 32, and past 64, points, with the last group ragged; in layer
runs and, with the ordinary kernels, in batches too large for runs.  Frontier and labels
removed equal the oracle's."""
import numpy as np
import pytest

import oracle
import pmdd_b200 as P
from pmdd_b200 import instances

KEYS = ("dominance_filtered_total",)
CASES = [(1, 5, 18), (1, 4, 26), (1, 7, 15), (2, 5, 70), (2, 4, 80)]


def diagram(ptype, d, n, seed):
    text = instances.knapsack_text(n, d, seed) if ptype == 1 else instances.setpacking_text(n, n // 5, d, seed)
    return P.DecisionDiagram.from_text(text, ptype, d)


def want(dd):
    st = {}
    pts = oracle.sorted_set(oracle.enumerate(dd, 1, state_dominance=1, stats=st))
    return pts, [int(st[k]) for k in KEYS]


@pytest.mark.parametrize("ptype,d,n", CASES)
def test_the_instances_have_such_nodes(ptype, d, n):
    pts, counts = want(diagram(ptype, d, n, 11 * n + d))
    assert len(pts) > 64 and counts[0] > 0


@pytest.mark.gpu
@pytest.mark.parametrize("ptype,d,n", CASES)
def test_state_dominance_of_many_labels(ptype, d, n):
    dds = [diagram(ptype, d, n, 11 * n + d + s) for s in range(2)]
    exp = [want(dd) for dd in dds]
    for dd, (pts, counts) in zip(dds, exp):
        st = {}
        got = P.enumerate_dd(dd, state_dominance=1, stats=st)
        assert np.array_equal(oracle.sorted_set(np.asarray(got, dtype=np.int64)), pts)
        assert [int(st[k]) for k in KEYS] == counts
    st = {}
    got = P.enumerate_batch(dds * 12, state_dominance=1, stats=st)
    for i, g in enumerate(got):
        assert np.array_equal(oracle.sorted_set(np.asarray(g, dtype=np.int64)), exp[i % 2][0])
    assert [int(st[k]) for k in KEYS] == [12 * (a + b) for a, b in zip(exp[0][1], exp[1][1])]
