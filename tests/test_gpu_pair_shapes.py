"""Which large FP32 grids step two steps per pass, and the columns of narrow ones.

Narrow grids (one column in x) have column shapes of their own; grids that
would leave most of every block idle, or have few planes, keep single steps.
Pulses, stubs and records are bitwise the single-step kernel's either way."""
import numpy as np
import pytest

from emsolver_b200.runner import build_solver, records
from tests.test_gpu_resident import small_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,per_pass", [
    (9, 1000, 130, 2),      # one column of 16 nodes, the second half of its row padding
    (16, 301, 227, 2),
    (27, 1013, 61, 2),      # one column of 32
    (33, 200, 170, 2),      # one column of 40
    (40, 181, 179, 2),
    (41, 173, 166, 2),      # two columns of the wider shapes
    (8, 400, 400, 1),
    (24, 24, 2000, 1),
    (1000, 1000, 2, 1),
    (500, 500, 5, 1),
    (7, 9, 20000, 1),
])
def test_narrow_and_flat_grids(built, nx, ny, nz, per_pass):
    w = small_grid(nx, ny, nz, 0.3, 21, (0, nx // 3, 2, 0.7))
    out = []
    for single in (True, False):
        s = build_solver(w, no_staging=single)
        s.step(5)
        s.step(w.steps - 5)
        assert s.stepsPerPass() == (1 if single else per_pass)
        out.append((s.pulses(), s.stubs(), records(s, w, f64=True)))
        s.close()
    assert np.abs(out[0][0]).max() > 0.0
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    for k in out[0][2]:
        assert np.array_equal(out[0][2][k], out[1][2][k]), k
