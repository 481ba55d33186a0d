"""FDTD grids whose columns would leave most of a block idle.

Long and flat grids run their sweeps in place on unpadded rows, others in one
pass on padded ones: every field value is that of the same step restated on the
host, float32 in the same order of operations."""
import numpy as np
import pytest

from emsolver_b200 import workloads
from emsolver_b200.fdtd import FIELDS, FdtdSolver
from emsolver_b200.solver import MatProps, TlmConfig, VoxelGridSpec

pytestmark = pytest.mark.gpu

EPS0, MU0, C0 = np.float32(8.8541878128e-12), np.float32(1.25663706212e-6), np.float32(299792458.0)


def host_steps(mat, table, dl, steps, source, amp):
    """E and H after `steps` steps, [z][y][x] arrays, a soft source in one cell (z polarised)."""
    f = np.float32
    nz, ny, nx = mat.shape
    dt = f(0.99) * f(dl) / (C0 * np.sqrt(f(3.0)))
    cmur = (C0 * dt - f(dl)) / (C0 * dt + f(dl))
    ch = dt / (MU0 * f(dl))
    ext = [(nz + 1, ny + 1, nx), (nz + 1, ny, nx + 1), (nz, ny + 1, nx + 1)]
    E = [np.zeros(s, f) for s in ext]
    H = [np.zeros(s, f) for s in [(nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)]]
    eps = np.ones(256, f)
    sig = np.zeros(256, f)
    for t, (e, s) in enumerate(table):
        eps[t + 2], sig[t + 2] = f(1) + (f(e) - f(1)), f(s)
    ca, cb, free = [], [], []
    for a in range(3):
        es, ss = np.zeros(ext[a], f), np.zeros(ext[a], f)
        cnt = np.zeros(ext[a], np.int32)
        pec = np.zeros(ext[a], bool)
        t1, t2 = [q for q in range(3) if q != a]          # x=0 y=1 z=2
        for d1 in (-1, 0):
            for d2 in (-1, 0):
                dst = [slice(None)] * 3
                for t, d in ((t1, d1), (t2, d2)):
                    n = mat.shape[2 - t]
                    dst[2 - t] = slice(1, n + 1) if d == -1 else slice(0, n)
                dst = tuple(dst)
                es[dst] += eps[mat]
                ss[dst] += sig[mat]
                cnt[dst] += 1
                pec[dst] |= mat == 1
        er, sg = es / cnt.astype(f), ss / cnt.astype(f)
        ep = EPS0 * np.maximum(f(1), er)
        lf = sg * dt / (f(2) * ep)
        ca.append((f(1) - lf) / (f(1) + lf))
        cb.append((dt / (ep * f(dl))) / (f(1) + lf))
        free.append(~pec)
    i, j, k = source
    for n in range(steps):
        for jj in (j, j + 1):
            for ii in (i, i + 1):
                if free[2][k, jj, ii]:
                    E[2][k, jj, ii] += (f(-0.25) * f(amp)) * SV[n]
        Ex, Ey, Ez = E
        H[0] -= ch * ((Ez[:, 1:, :] - Ez[:, :-1, :]) - (Ey[1:] - Ey[:-1]))
        H[1] -= ch * ((Ex[1:] - Ex[:-1]) - (Ez[:, :, 1:] - Ez[:, :, :-1]))
        H[2] -= ch * ((Ey[:, :, 1:] - Ey[:, :, :-1]) - (Ex[:, 1:, :] - Ex[:, :-1, :]))
        old = [e.copy() for e in E]
        Hx, Hy, Hz = H
        curl = [(Hz[1:-1, 1:, :] - Hz[1:-1, :-1, :]) - (Hy[1:, 1:-1, :] - Hy[:-1, 1:-1, :]),
                (Hx[1:, :, 1:-1] - Hx[:-1, :, 1:-1]) - (Hz[1:-1, :, 1:] - Hz[1:-1, :, :-1]),
                (Hy[:, 1:-1, 1:] - Hy[:, 1:-1, :-1]) - (Hx[:, 1:, 1:-1] - Hx[:, :-1, 1:-1])]
        inner = [np.s_[1:-1, 1:-1, :], np.s_[1:-1, :, 1:-1], np.s_[:, 1:-1, 1:-1]]
        for a in range(3):
            v = ca[a][inner[a]] * E[a][inner[a]] + cb[a][inner[a]] * curl[a]
            E[a][inner[a]] = np.where(free[a][inner[a]], v, f(0))
        for comp, ax in ((1, 0), (2, 0), (0, 1), (2, 1), (0, 2), (1, 2)):   # x, y, then z faces
            new, o = np.moveaxis(E[comp], 2 - ax, 0), np.moveaxis(old[comp], 2 - ax, 0)
            new[0] = o[1] + cmur * (new[1] - o[0])
            new[-1] = o[-2] + cmur * (new[-2] - o[-1])
    return E + H


SV = np.random.default_rng(4).standard_normal(64).astype(np.float32)


@pytest.mark.parametrize("nx,ny,nz", [(2, 3, 3000), (4, 4, 3000), (3, 300, 290), (5, 260, 250), (2, 500, 120), (7, 700, 40),
                                      (31, 30, 29)])
@pytest.mark.parametrize("dielectrics", [False, True])
def test_long_and_flat_grids(built, nx, ny, nz, dielectrics):
    rng = np.random.default_rng(nx + ny)
    mat = np.zeros((nz, ny, nx), np.uint8)
    if dielectrics:
        mat[nz // 4:nz // 2] = 2
        mat[:, ny // 3:ny // 2, nx // 2:] = 3
    mat[rng.random(mat.shape) < 0.02] = 1
    src = (nx // 2, ny // 2, nz // 2)
    mat[src[::-1]] = 0
    table = [(4.5, 0.05), (2.0, 0.0)] if dielectrics else []
    steps, dl = 40, 1e-3
    s = FdtdSolver()
    s.setup(VoxelGridSpec(nx, ny, nz, (0.0, 0.0, 0.0), dl), mat.reshape(-1), [MatProps(*t) for t in table],
            TlmConfig(f0=1e9, waveform=3, totalSteps=steps))
    s.setSourceTable(SV)
    cell = (src[2] * ny + src[1]) * nx + src[0]
    w = workloads.Workload("fd", nx, ny, nz, mat.reshape(-1), table, f0=1e9, waveform=3, steps=steps)
    assert w.cell(*src) == cell
    port = min(nx, ny) >= 3
    if port:
        s.addPort([cell], 2, 1.0)
    s.step(7)
    s.step(steps - 7)
    want = host_steps(mat, table, dl, steps, src, 1.0 if port else 0.0)
    assert (np.abs(want[2]).max() > 0.0) == port
    for k, r in zip(FIELDS, want):
        assert np.array_equal(s.field(k), r.reshape(-1)), k
    s.close()
