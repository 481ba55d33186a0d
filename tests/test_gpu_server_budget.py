"""A server whose budget holds a large request's state but no plan of two-step passes.

The request is admitted and steps one step per launch within the budget; with
more budget it may plan. Either way its results are bitwise the solve alone."""
import numpy as np
import pytest

from emsolver_b200 import Server, workloads
from emsolver_b200.runner import build_solver
from emsolver_b200.server import DONE, footprint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spare_bytes_per_node", [0, 40])
def test_budget_without_room_for_a_plan(built, spare_bytes_per_node):
    w = workloads.heterogeneous(n=104, steps=40)
    w.dft_freqs = np.array([1.0e9, 2.0e9])
    nodes = 104 ** 3
    state = (2 * 12 * 4 + 3 * 4 + 1) * nodes
    assert footprint(w) < state + (2 << 20)
    budget = state + (2 << 20) + spare_bytes_per_node * nodes
    with Server(hbm_budget=budget) as srv:
        rid = srv.submit(w)
        assert srv.wait(rid, 60.0) == DONE
        v, i, _ = srv.result(rid)
        assert srv.stats()["hbm_used_bytes"] == 0
    s = build_solver(w)
    s.step(w.steps)
    av, ai = s.portDft(0)
    s.close()
    assert np.array_equal(v, av) and np.array_equal(i, ai)
