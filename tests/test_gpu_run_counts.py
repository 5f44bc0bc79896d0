"""Layer runs (run.cu) and chains (chain.cu) take place and are counted apart: each call's
layers go to the counter of what expanded them, a run stops before the first oversized
destination and before a layer that outgrows a block, and the call goes on behind it."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import pmdd_b200 as P
from conftest import ROOT
from pmdd_b200 import instances

pytestmark = pytest.mark.gpu

RUN_BLOCKS, RUN_REGION, RESIDENT = 8, 2048, 1024


def one_node_a_layer(n, d, seed):
    """Items without weight and with profits of either sign: one node a layer, two arcs."""
    p = np.random.default_rng(seed).integers(-500, 501, size=(d, n))
    rows = [f"{n} 1 {d}"] + [" ".join(map(str, r)) for r in p] + [" ".join(["0"] * n) + " 1"]
    return "\n".join(rows) + "\n", p


CALLS = {
    "kp3": (1, lambda: instances.knapsack_text(20, 3, 3), 3, 1, 0),
    "kp3_sd": (1, lambda: instances.knapsack_text(20, 3, 3), 3, 1, 1),
    "sp3": (2, lambda: instances.setpacking_text(100, 20, 3, 37), 3, 1, 0),
    "sp3_sd": (2, lambda: instances.setpacking_text(91, 20, 3, 14), 3, 1, 1),
    "kp3_m3": (1, lambda: instances.knapsack_text(20, 3, 3), 3, 3, 0),
    "tsp3_m3": (3, lambda: instances.tsp_text(10, 3, 3), 3, 3, 0),
    "one_node": (1, lambda: one_node_a_layer(18, 4, 1)[0], 4, 1, 0),
    "kp1_wide": (1, lambda: instances.knapsack_text(60, 1, 5), 1, 1, 0),
}

CHILD = r"""
import json, sys
sys.path.insert(0, {root!r})
sys.path.insert(0, {tests!r})
import pmdd_b200 as P
from conftest import frontier_digest
from test_gpu_run_counts import CALLS
count = P._native.gpu_lib().pmdd_run_layer_count
out = {{}}
for name, (pt, text, d, method, sd) in CALLS.items():
    dd = P.DecisionDiagram.from_text(text(), pt, d)
    st, at = {{}}, count()
    got = P.enumerate_dd(dd, method=method, state_dominance=sd, stats=st)
    out[name] = [frontier_digest(got), st["layers_td"] + st["layers_bu"], count() - at, st["work_chained_layers"]]
print(json.dumps(out))
"""


def _run(**env):
    e = {k: v for k, v in os.environ.items() if not k.startswith(("PMDD_RUN_", "PMDD_CHAIN_"))}
    e.update(env)
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"))], env=e,
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr
    return json.loads(p.stdout.strip().splitlines()[-1])


@pytest.fixture(scope="module")
def default():
    return _run()


def test_runs_take_place_and_stop_where_they_should(default):
    for name in ("kp3", "kp3_sd"):
        _, layers, runs, chained = default[name]
        assert runs == layers == 20 and chained == 0, name
    for name in ("sp3_sd", "kp3_m3", "tsp3_m3"):
        _, layers, runs, chained = default[name]
        assert 0 < runs <= layers, name
    _, layers, runs, chained = default["sp3"]  # too wide in its middle: chains there
    assert runs > 0 and chained > 0 and runs + chained < layers

    # before the first destination of more than a tile's candidates
    _, p = one_node_a_layer(18, 4, 1)
    f, sizes = np.zeros((1, 4), dtype=np.int64), []
    for i in range(18):
        c = np.concatenate([f, f + p[:, i]])
        sizes.append(len(c))
        f = _maxima(c)
    first = next(i for i, s in enumerate(sizes) if s > RESIDENT)
    assert sizes[first] <= RUN_REGION  # the region would have held it
    assert default["one_node"][2] == first

    # before the first layer of which a block's share has too many arcs
    a = P.DecisionDiagram.from_text(CALLS["kp1_wide"][1](), 1, 1).arrays()
    lay, off = np.asarray(a["layer_offsets"]), np.asarray(a["in_arc_offsets"])

    def fits(y):
        n = lay[y + 1] - lay[y]
        cut = off[lay[y] + n * np.arange(RUN_BLOCKS + 1) // RUN_BLOCKS]
        return np.diff(cut).max() <= RUN_REGION and n <= RUN_BLOCKS * RUN_REGION

    first = next(y for y in range(1, len(lay) - 1) if not fits(y))
    _, layers, runs, _ = default["kp1_wide"]
    assert first - 1 <= runs < layers


def _maxima(c):
    c = np.unique(c, axis=0)
    ge = (c[None] >= c[:, None]).all(axis=2)
    np.fill_diagonal(ge, False)
    return c[~ge.any(axis=1)]


@pytest.mark.parametrize("env,runs,chains", [({"PMDD_RUN_LAYERS": "0"}, False, True),
                                             ({"PMDD_RUN_LAYERS": "3"}, True, True),
                                             ({"PMDD_CHAIN_LAYERS": "0"}, False, False)],
                         ids=["chains-alone", "short-runs", "neither"])
def test_each_counts_its_own_layers(env, runs, chains, default):
    got = _run(**env)
    for name, (digest, layers, r, c) in got.items():
        assert [digest, layers] == default[name][:2], name
        assert r + c <= layers, name
        if not runs:
            assert r == 0, name
        if not chains:
            assert c == 0, name
    assert (got["kp3"][2] > 0) == runs
    if chains and not runs:
        assert got["kp3"][3] > 0
    if chains:
        assert got["sp3"][3] > 0
