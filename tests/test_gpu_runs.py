"""Layer runs (run.cu): small layers of a request followed in one launch give the frontiers
and the work counters of the ordinary steps, by methods 1 and 3, whatever the run's length, for every
objective count, int32 and int64 points, with state dominance, from host and resident
DDs, and where a run stops at an oversized destination or a layer that outgrows a block."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import json, sys
sys.path.insert(0, {root!r})
sys.path.insert(0, {tests!r})
import numpy as np
import pmdd_b200 as P
from conftest import frontier_digest
from pmdd_b200 import instances as I
KEYS = ("work_candidates_total", "work_candidates_peak", "work_frontier_survivors_total",
        "work_frontier_peak_points", "dominance_filtered_total", "layers_td",
        "work_tile_candidates_total", "work_tile_survivors_total", "layers_bu", "layer_coupling", "cutset_size",
        "work_join_products_total")
out = []
def text(profits, weights, cap):
    rows = [f"{{profits.shape[1]}} 1 {{profits.shape[0]}}"] + [" ".join(map(str, r)) for r in profits]
    return "\n".join(rows + [" ".join(map(str, weights)) + f" {{cap}}"]) + "\n"
def add(call):
    st = {{}}
    res = call(st)
    out.append([[frontier_digest(r) if r.dtype == np.int32 else r[np.lexsort(r.T[::-1])].tolist() for r in res],
                [int(st[k]) for k in KEYS]])
for d in range(1, 9):
    n = 30 if d < 5 else 20
    add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(I.knapsack_text(n, d, 40 + d), 1, d), stats=st)])
p, w, c = I.knapsack_arrays(18, 3, 9)
add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(text(p.astype(np.int64) * 2_000_000, w, c), 1, 3), stats=st)])
p4, w4, c4 = I.knapsack_arrays(16, 4, 9)
add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(text(p4.astype(np.int64) * 2_000_000, w4, c4), 1, 4), stats=st)])
for pt, t, d in ((1, I.knapsack_text(40, 3, 5), 3), (1, I.knapsack_text(24, 4, 6), 4), (2, I.setpacking_text(91, 20, 3, 7), 3),
                 (2, I.setpacking_text(60, 20, 4, 8), 4), (3, I.tsp_text(10, 3, 1), 3), (3, I.tsp_text(9, 5, 2), 5)):
    for sd in (0, 1):
        add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(t, pt, d), state_dominance=sd, stats=st)])
        add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(t, pt, d), method=3, state_dominance=sd, stats=st)])
for d in range(1, 9):
    n = 30 if d < 5 else 20
    add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(I.knapsack_text(n, d, 80 + d), 1, d), method=3, stats=st)])
add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(text(p4.astype(np.int64) * 2_000_000, w4, c4), 1, 4), method=3,
                               stats=st)])
add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(I.tsp_text(3, 3, 1), 3, 3), method=3, stats=st)])
add(lambda st: [P.enumerate_dd(P.DecisionDiagram.from_text(I.knapsack_text(2, 3, 1), 1, 3), method=3, stats=st)])
res = P.ResidentSet.from_knapsack([I.knapsack_arrays(20 + i, 3, 60 + i) for i in range(5)])
add(lambda st: res.enumerate(stats=st))
add(lambda st: res.enumerate(state_dominance=1, stats=st))
tsp = P.ResidentSet.from_tsp([I.tsp_arrays(8 + i, 3, i) for i in range(3)])
add(lambda st: tsp.enumerate(stats=st))
add(lambda st: tsp.enumerate(method=3, stats=st))
add(lambda st: res.enumerate(method=3, stats=st))
add(lambda st: P.enumerate_batch([P.DecisionDiagram.from_text(I.knapsack_text(20 + i, 3 + i % 3, i), 1, 3 + i % 3)
                                  for i in range(12)], stats=st))
print(json.dumps(out))
"""


def _run(layers):
    e = dict(os.environ)
    e.pop("PMDD_RUN_LAYERS", None)
    if layers is not None:
        e["PMDD_RUN_LAYERS"] = str(layers)
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"))], env=e,
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr
    return json.loads(p.stdout.strip().splitlines()[-1])


@pytest.fixture(scope="module")
def without():
    return _run(0)


@pytest.mark.parametrize("layers", [1, 2, 7, None])
def test_runs_equal_ordinary_steps(layers, without):
    got = _run(layers)
    assert len(got) == len(without)
    for k, (a, b) in enumerate(zip(got, without)):
        assert a == b, k
