"""Short solves beside a long one, both in shared memory.

A handle on one thread steps many launch windows in one call while another one
steps a window per call on a second thread: the short calls take turns with the
long one's windows instead of waiting for all of them, and both results are
bitwise those of the single-step kernel."""
import threading

import numpy as np
import pytest

from emsolver_b200 import workloads
from emsolver_b200.runner import build_solver
from tests.test_gpu_resident import small_grid

pytestmark = pytest.mark.gpu

LONG, SHORT = 500, 20           # windows


def test_short_calls_take_turns(built):
    w = small_grid(64, 64, 60, 0.3, 64 * LONG, (0, 30, 1, 0.7))
    v = workloads.dipole(37, 31, 45, 11, steps=64 * SHORT)
    a, b = build_solver(w), build_solver(v)
    a.step(64)
    b.step(64)
    started, order, failed = threading.Event(), [], []

    def long():
        try:
            started.set()
            a.step(64 * (LONG - 1))
            order.append("long")
        except Exception as e:  # reported below
            failed.append(e)

    t = threading.Thread(target=long)
    t.start()
    started.wait()
    for _ in range(SHORT - 1):
        b.step(64)
    order.append("short")
    t.join()
    assert not failed and order == ["short", "long"]
    r = build_solver(v, no_staging=True)
    r.step(64 * SHORT)
    assert np.array_equal(b.pulses(), r.pulses())
    r = build_solver(w, no_staging=True)
    r.step(64 * LONG)
    assert np.array_equal(a.pulses(), r.pulses()) and np.array_equal(a.stubs(), r.stubs())
