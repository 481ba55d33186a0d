"""The allocation-free step uses the caller's stub planes on dielectric nodes only.

The stub planes hold NaN, infinities or large values on every other node (air,
PEC, row padding): pulses and the stubs of dielectric nodes are bitwise those
of a handle, and the other entries keep their bits. The grid has pairs of
nodes with the dielectric in front, behind and on both."""
import ctypes as C

import numpy as np
import pytest

from emsolver_b200 import MatProps, TlmConfig, TlmSolver, VoxelGridSpec, _lib
from tests.test_zz_no_alloc import connect, to_planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(9, 5, 4), (64, 31, 10)])
@pytest.mark.parametrize("junk", [np.nan, np.inf, -3e38, 1.0])
def test_stubs_of_other_nodes_are_not_used(built, nx, ny, nz, junk):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(nx)
    mat = np.zeros((nz, ny, nx), np.uint8)
    mat[rng.random(mat.shape) < 0.4] = 2
    mat[rng.random(mat.shape) < 0.05] = 1
    v0 = rng.standard_normal((nz, ny, nx, 12), dtype=np.float32)
    v0[mat == 1] = 0.0
    rho = np.float32(0.5)
    s = TlmSolver()
    s.setup(VoxelGridSpec(nx, ny, nz), mat.reshape(-1), [MatProps(4.5, 0.02)],
            TlmConfig(boundaryRho=float(rho), totalSteps=2, noStaging=True))
    s.setPulses(v0.reshape(-1))
    s.step(1)
    want = [s.pulses()]
    s.step(1)
    want.append(s.pulses())
    stubs, (yhat, ghat) = s.stubs(), s.tables()
    s.close()

    px = -(-nx // 8) * 8
    dev = torch.device("cuda", 0)
    padded = np.ones((nz, ny, px), np.uint8)
    padded[:, :, :nx] = mat
    a = torch.from_numpy(to_planes(v0.reshape(-1), nx, ny, nz).reshape(-1)).to(dev)
    b = torch.zeros_like(a)
    stub0 = np.broadcast_to(np.where(padded >= 2, np.float32(0), np.float32(junk)), (3, nz, ny, px)).copy()
    stub = torch.from_numpy(stub0).to(dev)
    dmat = torch.from_numpy(padded.reshape(-1)).to(dev)
    dy, dg = torch.from_numpy(yhat).to(dev), torch.from_numpy(ghat).to(dev)
    L = _lib.load()
    stream = C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
    for n, (src, dst) in enumerate([(a, b), (b, a)]):
        st = L.tlm_step_planes_noalloc(src.data_ptr(), dst.data_ptr(), stub.data_ptr(), dmat.data_ptr(),
                                       dy.data_ptr(), dg.data_ptr(), 1, nx, ny, nz, float(rho), 1 - n, None, stream)
        assert st == _lib.TLM_OK, L.tlm_last_error(None)
        torch.cuda.synchronize(dev)
        refl = dst.cpu().numpy().reshape(12, nz, ny, px)
        assert np.array_equal(connect(refl, padded, nx, ny, nz, rho), want[n])
    got = stub.cpu().numpy()
    diel = np.broadcast_to(padded >= 2, got.shape)
    assert np.array_equal(got[..., :nx].transpose(1, 2, 3, 0).reshape(-1)[np.repeat(mat.reshape(-1) >= 2, 3)],
                          stubs[np.repeat(mat.reshape(-1) >= 2, 3)])
    assert np.array_equal(got[~diel].view(np.uint32), stub0[~diel].view(np.uint32))
