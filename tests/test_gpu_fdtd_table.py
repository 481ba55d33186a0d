"""FDTD material tables longer than the 254 entries that a cell's byte can name.

The entries past those are read by no cell: fields and records bitwise the
same as with the first 254, or with only the ones in use."""
import numpy as np
import pytest

from emsolver_b200 import workloads
from emsolver_b200.fdtd import FdtdSolver
from emsolver_b200.solver import MatProps, TlmConfig, VoxelGridSpec

pytestmark = pytest.mark.gpu


def solve(mat, table, nx, ny, nz):
    s = FdtdSolver()
    s.setup(VoxelGridSpec(nx, ny, nz), mat.reshape(-1), table,
            TlmConfig(f0=workloads.gaussian_pulse_f0(1e-3, 6), waveform=2, totalSteps=12))
    s.addPlaneWave(0, 2, 2, 1.0)
    s.addProbe((4.5e-3, 4.5e-3, 4.5e-3))
    s.run()
    out = s.fields()
    out["probe"] = np.stack(s.probe(0))
    s.close()
    return out


@pytest.mark.parametrize("entries", [254, 255, 509, 510, 511, 600, 5000])
@pytest.mark.parametrize("used", [3, 254])
def test_long_tables(built, entries, used):
    nx, ny, nz = 19, 13, 11
    rng = np.random.default_rng(used)
    mat = rng.integers(2, 2 + used, (nz, ny, nx)).astype(np.uint8)
    mat[:, :, :5] = 0
    mat[0, 0, 0] = 1 + used
    props = [MatProps(float(e), float(g)) for e, g in zip(rng.uniform(1, 9, 5000), rng.uniform(0, 0.3, 5000))]
    want = solve(mat, props[:used], nx, ny, nz)
    got = solve(mat, props[:entries], nx, ny, nz)
    assert np.abs(want["Ez"]).max() > 0.0
    for k in want:
        assert np.array_equal(want[k], got[k]), k
