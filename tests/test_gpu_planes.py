"""The allocation-free step over caller-owned planes against a handle's step.

Both compute the same node updates in the same order: the state and the stubs
are compared bit for bit on grids from one node to several rounds of the
kernel's blocks, with PEC, walls and dielectrics or none; the energy is an FP64
sum of squares in another order, partial sums of a few thousand terms, so
relative 1e-12. Two calls in a row give the same energy bits (the last block to
finish adds the partials up in a fixed order and leaves its count at zero)."""
import ctypes as C

import numpy as np
import pytest

from emsolver_b200 import MatProps, TlmConfig, TlmSolver, VoxelGridSpec, _lib
from tests.test_zz_no_alloc import connect, to_planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (9, 2, 7), (64, 40, 33), (93, 80, 71), (120, 101, 60)])
@pytest.mark.parametrize("dielectrics", [False, True])
@pytest.mark.parametrize("rho", [0.5, -1.0])
def test_planes_step_equals_handle_step(built, nx, ny, nz, dielectrics, rho):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(nx + ny)
    mat = np.zeros((nz, ny, nx), np.uint8)
    if dielectrics:
        mat[rng.random(mat.shape) < 0.4] = 2
        mat[:, ny // 2:, :] = 3
    mat[rng.random(mat.shape) < 0.05] = 1
    table = [MatProps(4.5, 0.02), MatProps(2.0, 0.0)] if dielectrics else []
    v0 = rng.standard_normal((nz, ny, nx, 12), dtype=np.float32)
    v0[mat == 1] = 0.0
    s = TlmSolver()
    s.setup(VoxelGridSpec(nx, ny, nz), mat.reshape(-1), table, TlmConfig(boundaryRho=rho, totalSteps=1, noStaging=True))
    s.setPulses(v0.reshape(-1))
    s.step(1)
    want, energy = s.pulses(), s.getEnergyHistory(f64=True)[1][0]
    stubs, (yhat, ghat) = s.stubs(), s.tables()
    s.close()

    px = -(-nx // 8) * 8
    dev = torch.device("cuda", 0)
    a = torch.from_numpy(to_planes(v0.reshape(-1), nx, ny, nz).reshape(-1)).to(dev)
    b = torch.zeros_like(a)
    stub = torch.zeros((3, nz, ny, px), dtype=torch.float32, device=dev)
    padded = np.ones((nz, ny, px), np.uint8)
    padded[:, :, :nx] = mat
    dmat = torch.from_numpy(padded.reshape(-1)).to(dev)
    dy, dg = torch.from_numpy(yhat).to(dev), torch.from_numpy(ghat).to(dev)
    e = torch.zeros(2, dtype=torch.float64, device=dev)
    L = _lib.load()

    def call(slot):
        st = L.tlm_step_planes_noalloc(a.data_ptr(), b.data_ptr(), stub.data_ptr() if dielectrics else None,
                                       dmat.data_ptr(), dy.data_ptr() if dielectrics else None,
                                       dg.data_ptr() if dielectrics else None, len(table), nx, ny, nz, rho, 1,
                                       e.data_ptr() + 8 * slot, C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
        assert st == _lib.TLM_OK, L.tlm_last_error(None)

    call(0)
    torch.cuda.synchronize(dev)
    refl = b.cpu().numpy().reshape(12, nz, ny, px)
    assert np.array_equal(connect(refl, padded, nx, ny, nz, np.float32(rho)), want)
    assert np.all(refl[..., nx:] == 0.0)
    if dielectrics:
        got = stub.cpu().numpy()[..., :nx].transpose(1, 2, 3, 0).reshape(-1)
        assert np.array_equal(got, stubs)
    call(1)
    assert np.isclose(e[0].item(), energy, rtol=1e-12, atol=0.0)
    assert e[0].item() == e[1].item()
