"""The cutset join's rounds (couple.cu): a join whose survivors fit the buffer takes a seed and a
product round, one whose survivors outgrow it resumes, and either gives the oracle's frontier."""
import os
import re
import subprocess
import sys

import pytest

import oracle
import pmdd_b200 as P
from conftest import ROOT, frontier_digest
from pmdd_b200 import instances

pytestmark = pytest.mark.gpu

BUFFER = 1 << 17  # points, at least

CHILD = r"""
import sys
sys.path.insert(0, {root!r})
sys.path.insert(0, {tests!r})
import pmdd_b200 as P
from conftest import frontier_digest
from pmdd_b200 import instances
st = {{}}
dd = P.DecisionDiagram.from_text(instances.knapsack_text({n}, {d}, {seed}), 1, {d})
print(frontier_digest(P.enumerate_dd(dd, method=3, stats=st)), st["work_join_products_total"])
"""


@pytest.mark.parametrize("n,d,seed,resumes", [(20, 3, 3, False), (32, 5, 3, False), (50, 5, 1, True), (60, 4, 4000, True)])
def test_rounds_of_a_join(n, d, seed, resumes):
    env = dict(os.environ, PMDD_TRACE="1")
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"), n=n, d=d, seed=seed)],
                       env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    digest, products = p.stdout.split()
    rounds = len(re.findall(r"\[pmdd step\].* couple=1 ", p.stderr))
    assert int(products) > BUFFER or not resumes
    assert rounds > 2 if resumes else rounds == 2
    dd = P.DecisionDiagram.from_text(instances.knapsack_text(n, d, seed), 1, d)
    if n < 50:
        assert digest == frontier_digest(oracle.enumerate(dd, 3))
    else:  # tests of the two methods' agreement pin method 1 to the oracle
        assert digest == frontier_digest(P.enumerate_dd(dd, method=1))
