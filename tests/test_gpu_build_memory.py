"""Device memory of building and uploading sets: a knapsack set is built, and a set of diagrams
uploaded, in a budget that holds the diagrams and the construction's state arrays."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

BUILD = r"""
import sys
sys.path.insert(0, {root!r})
import numpy as np
import pmdd_b200 as P
from pmdd_b200 import instances
ks = [instances.knapsack_arrays(60, 2, 90 + i) for i in range({count})]
s = P.ResidentSet.from_knapsack(ks)
print(s.device_bytes, sum(s.dd_info(i)["num_nodes"] for i in range({count})))
"""

UPLOAD = r"""
import sys
sys.path.insert(0, {root!r})
import pmdd_b200 as P
from pmdd_b200 import instances
dd = P.DecisionDiagram.from_text(instances.knapsack_text(24, 2, 90), 1, 2)
s = P.ResidentSet([dd] * {count})
print(s.device_bytes)
"""


def _child(code, count, arena):
    env = dict(os.environ)
    env.pop("PMDD_ARENA_BYTES", None)
    if arena:
        env["PMDD_ARENA_BYTES"] = str(arena)
    return subprocess.run([sys.executable, "-c", code.format(root=ROOT, count=count)], env=env, capture_output=True,
                          text=True, timeout=300)


def test_knapsack_build_takes_no_more_than_the_diagrams_and_state_arrays():
    from pmdd_b200 import instances

    count = 6
    ks = [instances.knapsack_arrays(60, 2, 90 + i) for i in range(count)]
    state = sum(4 * (4 * 61 + 10) * (int(cap) + 1) for _, _, cap in ks)
    p = _child(BUILD, count, 0)
    assert p.returncode == 0, p.stderr
    nbytes, nodes = map(int, p.stdout.split())
    small = 64 * 1024 * count  # inputs, headers, descriptors, rounding
    assert small < 20 * nodes / 4 and nbytes + state > 80 << 20
    p = _child(BUILD, count, nbytes + state + small)
    assert p.returncode == 0, p.stderr


def test_upload_takes_no_more_than_the_diagrams():
    p = _child(UPLOAD, 1, 0)
    assert p.returncode == 0, p.stderr
    one = (int(p.stdout) + 255) // 256 * 256
    count = (80 << 20) // one + 1
    p = _child(UPLOAD, count, one * count)
    assert p.returncode == 0, p.stderr
