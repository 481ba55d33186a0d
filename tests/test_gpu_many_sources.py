"""More sources on a node pair than 16 bits count, on a grid that stays in shared memory.

33,000 plane waves through the same row put 66,000 entries on each of its
pairs; pulses and records are bitwise those of the single-step kernel."""
import numpy as np
import pytest

from emsolver_b200 import workloads
from emsolver_b200.runner import build_solver, records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waves", [32767, 32768, 33000])
def test_many_sources_on_one_pair(built, waves):
    w = workloads.Workload("waves", 4, 1, 3, np.zeros(12, np.uint8), [], waveform=2,
                           f0=workloads.gaussian_pulse_f0(1e-3, 6), steps=4, rho=0.3)
    w.probes_cell.append((1, 0, 1))
    out = []
    for single in (True, False):
        s = build_solver(w, no_staging=single)
        for q in range(waves):
            s.addPlaneWave(2, 1, q % 2, 1e-3 * (1 + q % 7))
        assert (s.stepsPerPass() > 1) != single
        s.step(w.steps)
        out.append((s.pulses(), records(s, w, f64=True)))
        s.close()
    assert np.abs(out[0][0]).max() > 0.0
    assert np.array_equal(out[0][0], out[1][0])
    for k in out[0][1]:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
