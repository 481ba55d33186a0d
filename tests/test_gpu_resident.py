"""Many steps per launch with the state in shared memory (small FP32 grids).

The resident kernel computes the same node updates in the same order as the
single-step kernel (tlm_config.no_staging = 1) and adds the energy shares up
in its order, so pulses, stubs, records and energies are compared bit for bit,
on grids that cut the bricks raggedly, from the smallest up to what the shared
memory holds, with PEC, walls, plane waves that put more entries into a brick
than it lists, launch windows of other lengths, and restored states. Two
handles on two threads run side by side."""
import threading

import numpy as np
import pytest

from emsolver_b200 import workloads
from emsolver_b200.runner import build_solver, records
from tests.test_gpu_pair import grid

pytestmark = pytest.mark.gpu


def small_grid(nx, ny, nz, rho, steps, wave):
    if min(nx, ny, nz) >= 5:
        w = grid(nx, ny, nz, rho, steps, seed=nx + ny)
    else:
        w = workloads.Workload("thin", nx, ny, nz, np.zeros(nx * ny * nz, np.uint8), [(3.0, 0.1)], waveform=2,
                               f0=workloads.gaussian_pulse_f0(1e-3, 6), steps=steps, rho=rho)
        w.mat[::7] = 2
        w.probes_cell += [(0, 0, 0), (nx - 1, ny - 1, nz - 1)]
    w.meta["plane_wave"] = wave
    return w


def run(w, single, restored, window=0):
    s = build_solver(w, no_staging=single, steps_per_launch=window)
    if not single:
        assert s.stepsPerPass() == min(window or 64, 64)
    if restored:
        v0 = np.random.default_rng(9).standard_normal(w.ncells * 12, dtype=np.float32)
        v0.reshape(-1, 12)[w.mat == 1] = 0.0
        s.setPulses(v0)
    s.step(5)
    s.step(w.steps - 5)
    out = s.pulses(), s.stubs(), records(s, w, f64=True)
    s.close()
    return out


def same(a, b):
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    for k in a[2]:
        assert np.array_equal(a[2][k], b[2][k]), k


@pytest.mark.parametrize("nx,ny,nz,rho,steps,wave", [
    (1, 1, 1, 0.3, 9, (0, 0, 2, 0.7)),
    (3, 2, 9, -1.0, 20, (2, 4, 0, 0.7)),
    (13, 9, 11, 0.0, 33, (0, 4, 2, 0.7)),
    (37, 31, 45, 0.3, 150, (2, 20, 0, 0.7)),   # a whole z plane of sources
    (61, 53, 47, 0.5, 70, (1, 7, 2, 0.7)),
    (64, 64, 64, 0.0, 40, (0, 30, 1, 0.7)),
    (200, 20, 19, 0.3, 20, (0, 66, 2, 0.7)),
    (8, 150, 40, 0.3, 40, (2, 3, 1, 0.7)),
    (500, 5, 7, -1.0, 20, (0, 66, 2, 0.7)),
])
@pytest.mark.parametrize("restored", [False, True])
def test_resident_equals_single_steps(built, nx, ny, nz, rho, steps, wave, restored):
    w = small_grid(nx, ny, nz, rho, steps, wave)
    same(run(w, True, restored), run(w, False, restored))


@pytest.mark.parametrize("window", [2, 7, 100])
def test_launch_windows(built, window):
    w = small_grid(37, 31, 45, 0.3, 130, (2, 20, 0, 0.7))
    same(run(w, True, False, window), run(w, False, False, window))


def test_two_threads(built):
    ws = [small_grid(64, 64, 60, 0.3, 400, (0, 30, 1, 0.7)), small_grid(61, 53, 47, 0.5, 400, (1, 7, 2, 0.7))]
    want = [run(w, True, False) for w in ws]
    got, failed = [None, None], []

    def work(i):
        try:
            for _ in range(3):
                got[i] = run(ws[i], False, False)
        except Exception as e:  # reported below
            failed.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for a, b in zip(want, got):
        same(a, b)
