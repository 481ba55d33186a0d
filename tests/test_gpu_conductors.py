"""Good conductors as materials: stub denominators from 2^24 to infinity.

The kernels that divide by a tabulated reciprocal (resident, two-step, planes)
against the single-step kernel, which divides as IEEE does: pulses and stubs
bit for bit, from states of ordinary size down to subnormal ones, whose
quotients lie where a rounded reciprocal would show."""
import ctypes as C

import numpy as np
import pytest

from emsolver_b200 import _lib
from emsolver_b200.runner import build_solver
from tests.test_gpu_pair import grid
from tests.test_zz_no_alloc import connect, to_planes

pytestmark = pytest.mark.gpu

SIGMA = [5.0e7, 1.0e9, 1.0e11, 1.0e13, 1.0e38, float("inf")]


def states(w):
    v0 = np.random.default_rng(9).standard_normal(w.ncells * 12, dtype=np.float32)
    v0.reshape(-1, 12)[w.mat == 1] = 0.0
    for power in (0, -70, -95, -120, -140):
        yield v0 * np.float32(2.0) ** power


@pytest.mark.parametrize("sigma", SIGMA)
@pytest.mark.parametrize("nx,ny,nz", [(37, 31, 45), (111, 101, 103)])
def test_kept_state_equals_single_steps(built, nx, ny, nz, sigma):
    w = grid(nx, ny, nz, 0.3, 4, seed=nx)
    w.table = [(4.5, sigma), (2.0, 0.02)]
    for v0 in states(w):
        out = []
        for single in (True, False):
            s = build_solver(w, no_staging=single)
            assert (s.stepsPerPass() > 1) != single
            s.setPulses(v0)
            s.step(1)
            s.step(w.steps - 1)
            out.append((s.pulses(), s.stubs()))
            s.close()
        assert np.isfinite(out[0][0]).all()
        assert np.array_equal(out[0][0], out[1][0])
        assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("sigma", SIGMA)
def test_planes_equal_single_steps(built, sigma):
    torch = pytest.importorskip("torch")
    nx, ny, nz = 40, 31, 10
    w = grid(nx, ny, nz, 0.3, 2, seed=nx)
    w.ports, w.probes_cell, w.meta = [], [], {}
    w.table = [(4.5, sigma), (2.0, 0.02)]
    dev = torch.device("cuda", 0)
    dmat = torch.from_numpy(w.mat).to(dev)
    L = _lib.load()
    for v0 in states(w):
        s = build_solver(w, no_staging=True)
        s.setPulses(v0)
        s.step(1)
        want, stubs, (yhat, ghat) = s.pulses(), s.stubs(), s.tables()
        s.close()
        a = torch.from_numpy(to_planes(v0, nx, ny, nz).reshape(-1)).to(dev)
        b = torch.zeros_like(a)
        stub = torch.zeros((3, nz, ny, nx), dtype=torch.float32, device=dev)
        dy, dg = torch.from_numpy(yhat).to(dev), torch.from_numpy(ghat).to(dev)
        st = L.tlm_step_planes_noalloc(a.data_ptr(), b.data_ptr(), stub.data_ptr(), dmat.data_ptr(), dy.data_ptr(),
                                       dg.data_ptr(), 2, nx, ny, nz, 0.3, 1, None,
                                       C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
        assert st == _lib.TLM_OK, L.tlm_last_error(None)
        torch.cuda.synchronize(dev)
        refl = b.cpu().numpy().reshape(12, nz, ny, nx)
        assert np.array_equal(connect(refl, w.mat.reshape(nz, ny, nx), nx, ny, nz, np.float32(0.3)), want)
        assert np.array_equal(stub.cpu().numpy().transpose(1, 2, 3, 0).reshape(-1), stubs)
