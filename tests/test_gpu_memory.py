"""Nearly full cards: optional scratch gives way, and what is read back needs little.

Two-step passes: with the card nearly full, reading the state needs more scratch than is left
beside the plan, and less than is left without it: the state is read all the
same, later steps run without a plan or with a new one, and everything is
bitwise what a handle with room gives. Where there is no room for a plan the
handle steps without one and holds nothing of it. FDTD fields are read in pieces
that fit what is left. A further handle takes back what others hold for speed alone (plans, second
field buffers). Each case runs in a process of
its own: the library's memory pool keeps what earlier handles had."""
import os
import subprocess
import sys

import numpy as np
import pytest

from emsolver_b200.runner import build_solver, records
from tests.test_gpu_pair import grid

pytestmark = pytest.mark.gpu

NX, NY, NZ = 304, 256, 256
MIB = 1 << 20


def fill(torch, leave):
    """Device memory taken until `leave` bytes are free."""
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


def state_read_beside_a_plan():
    import torch
    w = grid(NX, NY, NZ, 0.3, 10, seed=1)
    nodes = NX * NY * NZ
    state, plan = 48 * nodes, 18 * nodes
    out = []
    for tight in (True, False):
        s = build_solver(w)
        s.step(4)
        assert s.stepsPerPass() == 2
        hog = fill(torch, state - plan // 2) if tight else None
        got = [s.pulses(), s.stubs()]
        s.step(6)
        del hog
        torch.cuda.empty_cache()
        got += [s.pulses(), s.stubs(), records(s, w, f64=True)]
        s.close()
        out.append(got)
    for a, b in zip(out[0][:4], out[1][:4]):
        assert np.array_equal(a, b)
    for k in out[0][4]:
        assert np.array_equal(out[0][4][k], out[1][4][k]), k


def no_room_for_a_plan():
    import torch
    w = grid(NX, NY, NZ, 0.3, 6, seed=1)
    s = build_solver(w)
    s.step(1)                     # a single step: no plan yet
    before = s.deviceBytes()
    hog = fill(torch, 300 * MIB)
    s.step(3)
    assert s.stepsPerPass() == 1 and s.deviceBytes() == before
    del hog
    torch.cuda.empty_cache()
    got = s.pulses()
    s.close()
    r = build_solver(w)
    r.step(4)
    assert np.array_equal(got, r.pulses())
    r.close()


def field_read_on_a_full_card():
    import torch
    from emsolver_b200 import workloads
    from emsolver_b200.fdtd import FIELDS, build_fdtd
    small, large = workloads.heterogeneous(n=16, steps=3), workloads.heterogeneous(n=288, steps=3)
    s = build_fdtd(small)         # loads the kernels
    s.run()
    s.fields()
    s.close()
    s = build_fdtd(large)
    s.run()
    hog = fill(torch, 6 * MIB)
    got = s.fields()
    del hog
    torch.cuda.empty_cache()
    assert np.abs(got["Ez"]).max() > 0.0
    for k in FIELDS:              # in one piece or in others
        assert np.array_equal(got[k], s.field(k)), k
    s.close()


def second_handle_beside_a_plan():
    import torch
    nodes = NX * NY * NZ
    need, plan = (96 + 12 + 1) * nodes, 18 * nodes
    w = grid(NX, NY, NZ, 0.3, 6, seed=1)
    a = build_solver(w)
    a.step(3)
    assert a.stepsPerPass() == 2
    hog = fill(torch, need + 256 * MIB - plan // 2)
    b = build_solver(w)           # takes the plan's memory
    b.step(3)
    a.step(3)
    b.step(3)
    del hog                       # (reading the state needs 48 B per node)
    torch.cuda.empty_cache()
    got = [(s.pulses(), s.stubs()) for s in (a, b)]
    b.close()
    b = build_solver(w)
    b.step(6)
    for p, v in got:
        assert np.array_equal(p, b.pulses()) and np.array_equal(v, b.stubs())


def several_fdtd_handles():
    import torch
    from emsolver_b200 import workloads
    from emsolver_b200.fdtd import FIELDS, build_fdtd
    w = workloads.heterogeneous(n=320, steps=70)
    plane = 4 * 324 * 321 * 321
    build_fdtd(workloads.heterogeneous(n=16, steps=3)).run()
    hog = fill(torch, 4 * 13 * plane + 600 * MIB)
    s = [build_fdtd(w) for _ in range(4)]    # 13 planes each, the first two with six more until others need them
    for q in s:
        q.step(3)
    s.pop(0).close()
    s.pop(0).close()
    for q in s:                              # with room again
        q.step(67)
    got = [q.fields() for q in s]
    del hog, s
    torch.cuda.empty_cache()
    r = build_fdtd(w)
    r.run()
    want = r.fields()
    assert np.abs(want["Ez"]).max() > 0.0
    for g in got:
        for k in FIELDS:
            assert np.array_equal(g[k], want[k]), k


@pytest.mark.parametrize("case", ["second_handle_beside_a_plan", "several_fdtd_handles", "field_read_on_a_full_card", "state_read_beside_a_plan", "no_room_for_a_plan"])
def test_nearly_full_card(built, case):
    pytest.importorskip("torch")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", f"from tests import test_gpu_memory as t; t.{case}()"], cwd=root,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
