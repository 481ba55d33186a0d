"""The staged FP32 kernel itself, and what asks for it.

Single FP32 steps run their interior tiles staged on grids of 2^20 padded nodes
and more, and on smaller ones where a stage wait limit is given: pulses,
stubs, records and surface monitors bitwise those of the single kernel with
direct loads and of the oracle, with every step a staged one. A limit that
runs out fails the call, also where it asks for several steps at once."""
import numpy as np
import pytest

from emsolver_b200 import _lib, workloads
from emsolver_b200.runner import build_solver, records
from oracle import Oracle, drive
from tests.golden.cases import mid_cases, staged_tiles, stub_tile_counts
from tests.test_gpu_interior import slab_dipole

pytestmark = pytest.mark.gpu

LIMIT_US = 2_000_000


def staged_solver(w, **kw):
    s = build_solver(w, **kw)
    assert staged_tiles(w) > 0 and s.stepLaunches() >= 2
    return s


def same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("case", ["heterogeneous", "mid", "air_odd"])
def test_staged_equals_direct_loads_and_oracle(built, case):
    w = workloads.heterogeneous(n=64, steps=30) if case == "heterogeneous" else \
        mid_cases()[0] if case == "mid" else slab_dipole()
    if case != "mid":
        assert stub_tile_counts(w)[0] > 0
    s, r = staged_solver(w, stage_wait_us=LIMIT_US), build_solver(w, no_staging=True)
    assert s.stepsPerPass() == 1 and r.stepLaunches() == 1
    s.step(w.steps)
    r.step(w.steps)
    O = Oracle(False)
    drive.setup(O, w)
    drive.advance(O, w, w.steps)
    assert np.array_equal(s.pulses(), r.pulses()) and np.array_equal(s.pulses(), O.pulses())
    if w.table:
        assert np.array_equal(s.stubs(), r.stubs()) and np.array_equal(s.stubs(), O.stubs())
    same(records(s, w, f64=True), records(r, w, f64=True))


def test_large_grid_step_by_step(built):
    w = workloads.heterogeneous(n=104, steps=18, seed=3)
    s, r = staged_solver(w), build_solver(w, no_staging=True)
    for _ in range(w.steps):
        s.step(1)
    r.step(w.steps)
    assert np.array_equal(s.pulses(), r.pulses()) and np.array_equal(s.stubs(), r.stubs())
    same(records(s, w, f64=True), records(r, w, f64=True))


def test_large_grid_with_surface_monitors(built):
    w = workloads.dipole(112, 104, 97, 21, slab=(9, 40, 3.0), steps=130, name="monitored")
    w.meta.update(surface_monitors=True, huy_offset=8, settle_steps=60, field_plane=(1, 50), record_every=16)
    out = []
    for s in (staged_solver(w), build_solver(w, no_staging=True)):
        assert s.stepsPerPass() == 1
        s.step(w.steps)
        mag, re, im, _ = s.getJsDft(raw=True)
        got = records(s, w, f64=True)
        got.update(js=s.getJsInstant(), mag=mag, re=re, im=im, huy=s.huygensDft()[0], plane=s.getFieldPlane()[0],
                   frames=np.stack([s.getFrame(i)["js"] for i in range(s.frameCount())]), far=s.computeFarField(7, 13)["U"],
                   pulses=s.pulses(), stubs=s.stubs())
        out.append(got)
        s.close()
    assert np.abs(out[0]["huy"]).max() > 0.0
    same(*out)


@pytest.mark.parametrize("n", [40, 104])
def test_limit_that_runs_out(built, n):
    w = workloads.heterogeneous(n=n, steps=24)
    s = build_solver(w, stage_wait_us=-1)
    with pytest.raises(_lib.TlmError) as err:
        s.step(w.steps)
    assert err.value.status == _lib.TLM_ECUDA and "never arrived" in str(err.value)
    s.close()
    s, r = build_solver(w), build_solver(w, no_staging=True)
    s.step(w.steps)
    r.step(w.steps)
    assert np.array_equal(s.pulses(), r.pulses())
