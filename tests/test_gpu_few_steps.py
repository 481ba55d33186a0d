"""Small grids stepped a few steps per call.

Calls of one to a few steps, whichever of the resident and the single-step
kernels they take, leave bitwise the state, stubs and records of one call, on
grids with one and with two node pairs per thread."""
import numpy as np
import pytest

from emsolver_b200.runner import build_solver, records
from tests.test_gpu_resident import small_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(37, 31, 45), (61, 53, 47), (64, 64, 64), (500, 10, 10)])
def test_calls_of_a_few_steps(built, nx, ny, nz):
    calls = [1, 2, 3, 4, 5, 2, 63, 64, 3, 65, 66, 67, 68]
    w = small_grid(nx, ny, nz, 0.3, sum(calls), (0, nx // 2, 1, 0.7))
    out = []
    for few in (True, False):
        s = build_solver(w, no_staging=not few)
        for n in calls if few else [sum(calls)]:
            s.step(n)
        out.append((s.pulses(), s.stubs(), records(s, w, f64=True)))
        s.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    for k in out[0][2]:
        assert np.array_equal(out[0][2][k], out[1][2][k]), k
