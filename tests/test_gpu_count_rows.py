"""The count kernel's rows: diagrams whose layers' arcs and destinations lie on both sides of
one short row (1024), of four destination rows (4096) and of a full arc row (8192) give the
oracle's frontier, candidates and survivors, with host steps and chained, by methods 1
and 3."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
import pmdd_b200 as P
from conftest import ROOT
from pmdd_b200 import instances

CASES = [(1, 1, 60), (1, 2, 44), (3, 1, 12)]
CHILD = r"""
import sys
sys.path.insert(0, {root!r})
sys.path.insert(0, {root!r} + "/tests")
import numpy as np
import oracle
import test_gpu_count_rows as M
for c in M.CASES:
    M.check(*c)
"""


def diagram(ptype, d, n):
    text = instances.knapsack_text(n, d, 5 + n) if ptype == 1 else instances.tsp_text(n, d, 5 + n)
    return P.DecisionDiagram.from_text(text, ptype, d)


def check(ptype, d, n):
    dd = diagram(ptype, d, n)
    ost = {}
    want = oracle.sorted_set(oracle.enumerate(dd, 1, stats=ost))
    for method in (1, 3):
        st = {}
        got = P.enumerate_dd(dd, method=method, stats=st)
        assert np.array_equal(oracle.sorted_set(np.asarray(got, dtype=np.int64)), want), (ptype, d, n, method)
        if method == 1:
            assert st["work_candidates_total"] == ost["candidates_total"]
            assert st["work_frontier_survivors_total"] == ost["survivors_total"]


def test_the_layers_lie_on_both_sides():
    arcs, nodes = set(), set()
    for c in CASES:
        a = diagram(*c).arrays()
        lay = np.asarray(a["layer_offsets"])
        arcs |= set(np.diff(np.asarray(a["in_arc_offsets"])[lay]).tolist())
        nodes |= set(np.diff(lay).tolist())
    for lo, hi in ((1, 1024), (1025, 8192), (8193, 9216), (9217, 1 << 30)):
        assert any(lo <= x <= hi for x in arcs), (lo, hi)
    for lo, hi in ((1, 1024), (1025, 4096), (4097, 1 << 30)):
        assert any(lo <= x <= hi for x in nodes), (lo, hi)


@pytest.mark.gpu
@pytest.mark.parametrize("chain", ["0", "8"])
def test_counts_of_wide_layers(chain):
    e = dict(os.environ, PMDD_CHAIN_LAYERS=chain, PMDD_RUN_LAYERS="0")
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=e, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr
