"""Layer runs and device memory: an allocation that fails for a run, or in the step that has
one, costs the run and not the request (it goes on by ordinary steps)."""
import numpy as np
import pytest

import oracle
import pmdd_b200 as P
from pmdd_b200 import instances

pytestmark = pytest.mark.gpu

# (problem type, method, state dominance, allocations of the admission, of the run and its step)
CASES = [(1, 1, 0, 2, 2 + 1 + 2), (1, 1, 1, 2, 2 + 1 + 2), (2, 1, 1, 2, 2 + 1 + 2), (1, 3, 0, 3, 4 + 2 + 2)]


@pytest.mark.parametrize("ptype,method,sd,admission,step", CASES)
def test_one_failed_allocation_costs_the_run_only(ptype, method, sd, admission, step, monkeypatch):
    monkeypatch.setenv("PMDD_SERVER_LANES", "1")
    monkeypatch.delenv("PMDD_RUN_LAYERS", raising=False)
    text = instances.knapsack_text(14, 3, 5) if ptype == 1 else instances.setpacking_text(40, 20, 3, 5)
    dd = P.DecisionDiagram.from_text(text, ptype, 3)
    want = oracle.sorted_set(oracle.enumerate(dd, method))
    for after in range(admission, admission + step):
        srv = P.Server(budget_bytes=1 << 30)
        try:
            assert srv.submit(dd, 7, method=method, state_dominance=sd) == 0
            srv.inject_alloc_failures(after, 1)
            srv.run(0)
            r = srv.poll()
            assert srv.info()["injected_alloc_failures"] == 1, after
        finally:
            srv.close()
        assert r is not None and r.status == 0, (after, r and r.error)
        assert np.array_equal(oracle.sorted_set(r.frontier), want), after
