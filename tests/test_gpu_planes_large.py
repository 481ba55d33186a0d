"""The allocation-free step on grids of several waves of blocks.

A block walks over one tile or several, by the size and by whether an energy is
asked for: pulses of an incident and of a reflected input are the same bits
with and without one, those of the handle's step, and the energy is within
1e-12 of its (an FP64 sum of squares in another order)."""
import ctypes as C

import numpy as np
import pytest

from emsolver_b200 import TlmConfig, TlmSolver, VoxelGridSpec, _lib
from tests.test_zz_no_alloc import connect, to_planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(96, 80, 79), (104, 96, 62), (128, 130, 130), (163, 161, 160), (200, 205, 203)])
def test_waves_of_blocks(built, nx, ny, nz):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(nx)
    mat = np.zeros((nz, ny, nx), np.uint8)
    mat[rng.random(mat.shape) < 0.01] = 1
    v0 = rng.standard_normal((nz, ny, nx, 12), dtype=np.float32)
    v0[mat == 1] = 0.0
    rho = np.float32(0.5)
    s = TlmSolver()
    s.setup(VoxelGridSpec(nx, ny, nz), mat.reshape(-1), [], TlmConfig(boundaryRho=0.5, totalSteps=1, noStaging=True))
    s.setPulses(v0.reshape(-1))
    s.step(1)
    want, energy = s.pulses(), s.getEnergyHistory(f64=True)[1][0]
    s.close()
    px = -(-nx // 8) * 8
    dev = torch.device("cuda", 0)
    padded = np.ones((nz, ny, px), np.uint8)
    padded[:, :, :nx] = mat
    dmat = torch.from_numpy(padded.reshape(-1)).to(dev)
    a = torch.from_numpy(to_planes(v0.reshape(-1), nx, ny, nz).reshape(-1)).to(dev)
    b, c, d = (torch.full_like(a, float("nan")) for _ in range(3))
    e = torch.zeros(2, dtype=torch.float64, device=dev)
    L = _lib.load()
    stream = C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)

    def call(src, dst, incident, slot):
        st = L.tlm_step_planes_noalloc(src.data_ptr(), dst.data_ptr(), None, dmat.data_ptr(), None, None, 0, nx, ny, nz,
                                       0.5, incident, e.data_ptr() + 8 * slot if slot is not None else None, stream)
        assert st == _lib.TLM_OK, L.tlm_last_error(None)

    call(a, b, 1, 0)
    call(a, c, 1, None)
    assert torch.equal(b, c)
    call(b, c, 0, 1)
    call(b, d, 0, None)
    assert torch.equal(c, d)
    refl = b.cpu().numpy().reshape(12, nz, ny, px)
    inc = connect(refl, padded, nx, ny, nz, rho)
    assert np.array_equal(inc, want)
    assert np.isclose(e[0].item(), energy, rtol=1e-12, atol=0.0)
    assert np.isclose(e[1].item(), np.square(inc, dtype=np.float64).sum(), rtol=1e-12, atol=0.0)
