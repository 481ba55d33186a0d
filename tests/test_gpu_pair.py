"""Two steps per pass over memory (FP32 grids of 2^20 padded nodes and more).

The pass computes the same node updates in the same order as two single
steps, so pulses, stubs, probe and port records are compared bit for bit: with
the single-step kernel (tlm_config.no_staging = 1) on grids whose sizes cut the
columns and plane ranges raggedly, and with the oracle. The energy is an FP64
sum of squares, on the device in the order of the single-step tiles, in the
oracle in another: partial sums of at most a few thousand terms each, so
relative 1e-12."""
import numpy as np
import pytest

from emsolver_b200 import workloads
from emsolver_b200.runner import build_solver, records
from emsolver_b200.workloads import Workload
from oracle import Oracle, drive

pytestmark = pytest.mark.gpu

ENERGY_RTOL = 1e-12


def grid(nx, ny, nz, rho, steps, seed):
    """Two lossy boxes, scattered PEC and a PEC wall, three ports (one per
    axis), probes inside and in two corners, a plane-wave source."""
    rng = np.random.default_rng(seed)
    mat = np.zeros((nz, ny, nx), np.uint8)
    mat[nz // 5:nz // 2, ny // 6:ny // 2 + 1, nx // 4:nx - nx // 5] = 2
    mat[nz // 3:nz - 2, ny // 2:, :nx // 2] = 3
    mat[rng.random((nz, ny, nx)) < 0.003] = 1
    mat[nz // 2:nz // 2 + 3, :, nx - 4:] = 1
    w = Workload("pair", nx, ny, nz, mat.reshape(-1), [(4.5, 0.02), (2.0, 0.0)],
                 f0=workloads.gaussian_pulse_f0(1e-3, 6), waveform=2, steps=steps, rho=rho)
    for pol in range(3):
        while True:
            c = [int(rng.integers(2, v - 2)) for v in (nx, ny, nz)]
            if mat[c[2], c[1], c[0]] == 0:
                break
        w.ports.append(([w.cell(*c)], pol, 1.0 + pol))
    for _ in range(4):
        w.probes_cell.append(tuple(int(rng.integers(0, v)) for v in (nx, ny, nz)))
    w.probes_cell += [(0, 0, 0), (nx - 1, ny - 1, nz - 1)]
    w.meta["plane_wave"] = (0, nx // 3, 2, 0.7)
    return w


def compare(a, b):
    for k in a:
        if k == "energy":
            assert np.allclose(a[k], b[k], rtol=ENERGY_RTOL, atol=0.0)
        else:
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("nx,ny,nz,rho,steps", [
    (111, 101, 103, 0.3, 37),     # nothing divides anything; odd nx, a step left over
    (128, 128, 128, 0.0, 66),     # crosses a launch window
    (97, 230, 61, -1.0, 21),
    (1040, 64, 17, 0.5, 18),      # many columns in x, thin in z
    (16, 400, 200, 0.3, 19),      # one column in x
    (40, 27, 1200, 0.3, 19),      # long in z
])
@pytest.mark.parametrize("restored", [False, True])
def test_pass_equals_two_steps(built, nx, ny, nz, rho, steps, restored):
    """From zero fields (most numerators zero, tiny or subnormal) and from a
    random state."""
    w = grid(nx, ny, nz, rho, steps, seed=nx)
    out = []
    for single in (True, False):
        s = build_solver(w, no_staging=single)
        assert s.stepsPerPass() == (1 if single else 2)
        if restored:
            v0 = np.random.default_rng(9).standard_normal(w.ncells * 12, dtype=np.float32)
            v0.reshape(-1, 12)[w.mat == 1] = 0.0
            s.setPulses(v0)
        s.step(5)
        s.step(steps - 5)
        out.append((s.pulses(), s.stubs(), records(s, w, f64=True)))
        s.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    compare(out[0][2], out[1][2])


def test_pass_equals_oracle(built):
    w = workloads.heterogeneous(n=104, steps=12, seed=3)
    s = build_solver(w)
    assert s.stepsPerPass() == 2
    s.step(w.steps)
    O = Oracle(False)
    drive.setup(O, w)
    drive.advance(O, w, w.steps)
    assert np.array_equal(s.pulses(), O.pulses())
    assert np.array_equal(s.stubs(), O.stubs())
    ra, ro = records(s, w), drive.records(O, w)
    for k in ra:
        if not k.startswith("energy"):
            assert np.array_equal(ra[k], ro[k]), k
