"""When a large FP32 handle plans its two-step passes.

A plan takes as long as several steps: handles that are asked for fewer keep
single steps and hold no plan's memory, a host that steps little by little
plans in the end, and the results are bitwise the same."""
import numpy as np
import pytest

from emsolver_b200.runner import build_solver
from tests.test_gpu_pair import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calls,planned", [([3], False), ([2, 2], False), ([64], True), ([2] * 40, True)])
def test_few_steps_do_not_plan(built, calls, planned):
    w = grid(104, 104, 104, 0.3, sum(calls), seed=5)
    s, r = build_solver(w), build_solver(w, no_staging=True)
    s.step(1)
    r.step(1)
    before = s.deviceBytes()
    for n in calls:
        s.step(n)
    r.step(sum(calls))
    assert (s.deviceBytes() > before + 4 * 104 ** 3) == planned
    assert s.stepsPerPass() == 2
    assert np.array_equal(s.pulses(), r.pulses()) and np.array_equal(s.stubs(), r.stubs())
    s.close()
    r.close()
