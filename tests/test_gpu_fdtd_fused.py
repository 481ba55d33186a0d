"""The FDTD step in one pass over memory against the in-place sweeps.

The fused pass (and its Mur kernel) computes the same updates in the same order
as the in-place H and E sweeps (tlm_config.no_staging = 1, which the golden
vectors of the reference also pin through the default path), so every field
value, port and probe record is compared bit for bit; the energy sums the same
arrays in the same order, so it is equal too. Sizes cut the columns and plane
ranges raggedly, down to the smallest grid; tables with many materials overflow
the coefficient table, so that edges read theirs one by one."""
import numpy as np
import pytest

from emsolver_b200 import workloads
from emsolver_b200.fdtd import FIELDS, FdtdSolver
from emsolver_b200.solver import MatProps, TlmConfig, VoxelGridSpec

pytestmark = pytest.mark.gpu


def solve(nx, ny, nz, materials, in_place, steps=23):
    rng = np.random.default_rng(nx * 7 + ny * 3 + nz)
    mat = np.zeros((nz, ny, nx), np.uint8)
    if materials == 3:
        mat[nz // 5:nz // 2, ny // 6:ny // 2 + 1, nx // 4:nx - nx // 5] = 2
        mat[nz // 3:nz - 1, ny // 2:, :nx // 2] = 3
        mat[:, 0:2, :] = 4
    elif materials:
        mat[...] = rng.integers(2, 2 + materials, mat.shape)
    mat[rng.random(mat.shape) < 0.02] = 1
    table = [MatProps(float(rng.uniform(1.0, 9.0)), float(rng.uniform(0.0, 0.3))) for _ in range(materials)]
    c = (nx // 2, ny // 2, nz // 2)
    port = min(nx, ny, nz) >= 3
    mat[c[2], c[1], c[0]] = 0
    s = FdtdSolver()
    s.setup(VoxelGridSpec(nx, ny, nz), mat.reshape(-1), table,
            TlmConfig(f0=workloads.gaussian_pulse_f0(1e-3, 6), waveform=2, totalSteps=steps, noStaging=in_place))
    if port:
        s.addPort([(c[2] * ny + c[1]) * nx + c[0]], 2, 1.0)
    s.addPlaneWave(0, max(1, nx // 3), 2, 0.7)
    s.addProbe(tuple((v + 0.5) * 1e-3 for v in c))
    s.addProbe((0.5e-3, 0.5e-3, 0.5e-3))
    s.step(4)
    s.step(steps - 4)
    out = {k: s.field(k) for k in FIELDS}
    out["energy"] = s.getEnergyHistory(f64=True)[1]
    for q in range(2):
        out[f"probe{q}"] = np.stack(s.probe(q))
    if port:
        out["port"] = np.stack(s.port(0))
    s.close()
    return out


@pytest.mark.parametrize("materials", [0, 3, 40])
@pytest.mark.parametrize("nx,ny,nz", [(2, 2, 2), (3, 5, 9), (17, 19, 23), (65, 66, 67), (101, 64, 33), (203, 31, 18),
                                      (30, 140, 21), (20, 22, 150)])
def test_fused_pass_equals_in_place_sweeps(built, nx, ny, nz, materials):
    a, b = (solve(nx, ny, nz, materials, in_place) for in_place in (True, False))
    assert np.abs(a["Ez"]).max() > 0.0
    for k in a:
        assert np.array_equal(a[k], b[k]), k
