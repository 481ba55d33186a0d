"""Timed cases: what a user of this library has it do, through its public calls.

Six kinds of work, over the sizes that the workloads module, the tests and the
benchmark use:

solve      a whole TLM solve: set up a grid from a host material map, run its
           steps, read back port and probe records, port DFT and energy
resume     a checkpointed TLM state put back into a kept handle, advanced, and
           read back whole (pulses and stubs)
far_field  a TLM antenna solve with surface currents, a Huygens box and the
           far-field transform
batch      many TLM solves of different sizes advanced together
planes     one TLM step over device planes that the caller owns
fdtd       a whole Yee FDTD solve with its records

`exact` restates each of them in 64 bits with plain torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from emsolver_b200 import _lib, workloads
from emsolver_b200.batch import Batch
from emsolver_b200.fdtd import build_fdtd
from emsolver_b200.runner import build_solver
from emsolver_b200.solver import Storage
from emsolver_b200.workloads import Workload

STORAGES = {"f32": Storage.F32, "f64": Storage.F64, "f16": Storage.F16, "bf16": Storage.BF16,
            "bfp16": Storage.BFP16}
BYTES = {"f32": 4, "f64": 8, "f16": 2, "bf16": 2, "bfp16": 2}


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # a small antenna, odd in every direction, solved on its own: every
        # step is a few microseconds of work, so launches and latency count;
        # its final pulses are kept for a later restart
        dict(name="dipole_small", kind="solve", scene="dipole", nx=37, ny=31, nz=45, storage="f32", steps=1000,
             rho=0.0, near_field=0, state=True),
        # the 64^3 free-space pulse that the tests pin (500 steps)
        dict(name="free_space_64", kind="solve", scene="free", nx=64, ny=64, nz=64, storage="f32", steps=500,
             rho=0.0, near_field=0),
        # the benchmark's grid: 16 lossy dielectric boxes, 8 probes
        dict(name="hetero_192", kind="solve", scene="hetero", nx=192, ny=192, nz=192, storage="f32", steps=256,
             rho=0.0, near_field=0),
        # the largest: an antenna in 37.7 M cells
        dict(name="dipole_large", kind="solve", scene="dipole", nx=384, ny=384, nz=256, storage="f32", steps=96,
             rho=0.0, near_field=0),
        # 16-bit storage with the exact box around the antenna, ragged sizes
        dict(name="dipole_f16", kind="solve", scene="dipole", nx=251, ny=237, nz=190, storage="f16", steps=128,
             rho=0.0, near_field=6),
        # the double-precision mode, partly reflecting walls
        dict(name="hetero_f64", kind="solve", scene="hetero", nx=118, ny=101, nz=96, storage="f64", steps=128,
             rho=0.3, near_field=0),
        # block floating point on a mid-size lossy grid
        dict(name="hetero_bfp16", kind="solve", scene="hetero", nx=160, ny=144, nz=128, storage="bfp16", steps=192,
             rho=0.0, near_field=0),
        # a saved state carried on: PEC cells, dielectrics, reflecting walls
        dict(name="resume_odd", kind="resume", nx=61, ny=53, nz=47, steps=64, rho=0.3),
        # an antenna's radiation pattern
        dict(name="far_field_96", kind="far_field", nx=104, ny=96, nz=101, steps=160, huy=10, ntheta=37, nphi=73),
        # a parameter study: dipoles with edges of 24 to 96 cells
        dict(name="batch_48", kind="batch", count=48, lo=24, hi=96, steps=200),
        # one step inside a host program that keeps the planes itself
        dict(name="planes_odd", kind="planes", nx=93, ny=80, nz=71, rho=0.5),
        # the Yee solver on the benchmark's grid
        dict(name="fdtd_192", kind="fdtd", scene="hetero", nx=192, ny=192, nz=192, steps=384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "resume", "far_field", "batch", "planes", "fdtd", "fdtd"])
    if kind == "batch":
        lo = rng.randint(20, 40)
        return dict(kind=kind, count=rng.randint(8, 48), lo=lo, hi=lo + rng.randint(16, 56),
                    steps=rng.randint(60, 220))
    if kind == "planes":
        nx, ny, nz = (_log_int(rng, 14, 200) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, rho=rng.choice([0.0, 0.3, 0.5, -1.0]))
    if kind == "resume":
        nx, ny, nz = (_log_int(rng, 16, 90) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randint(9, 96), rho=rng.choice([0.0, 0.3, -1.0]))
    if kind == "far_field":
        nx, ny, nz = (_log_int(rng, 48, 150) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randint(60, 160), huy=rng.randint(4, 10),
                    ntheta=rng.choice([19, 37]), nphi=rng.choice([37, 73]))
    cells = math.exp(rng.uniform(math.log(2.5e4), math.log(1.2e7)))
    edge = cells ** (1.0 / 3.0)
    fx, fy = rng.uniform(0.75, 1.35), rng.uniform(0.75, 1.35)
    nx, ny = max(17, int(edge * fx)), max(17, int(edge * fy))
    nz = max(17, int(cells / (nx * ny)))
    steps = int(min(1000, max(48, 1.2e9 / (nx * ny * nz)))) - rng.randint(0, 17)
    if kind == "fdtd":
        return dict(kind=kind, scene=rng.choice(["hetero", "dipole"]), nx=nx, ny=ny, nz=nz, steps=steps)
    storage = rng.choice(["f32", "f32", "f32", "f32", "f64", "f16", "bf16", "bfp16"])
    scene = rng.choice(["free", "hetero", "dipole", "dipole"])
    near = rng.choice([0, 6]) if storage in ("f16", "bf16") and scene == "dipole" else 0
    return dict(kind="solve", scene=scene, nx=nx, ny=ny, nz=nz, storage=storage, steps=steps,
                rho=rng.choice([0.0, 0.0, 0.3, -1.0]), near_field=near,
                state=cells < 1e5 and storage in ("f32", "f64"))


# ---------------------------------------------------------------- the grids

def _hetero(nx, ny, nz, steps, seed):
    """The benchmark's scene on a box of any size: 16 lossy boxes, a
    differentiated-Gaussian port on an air cell, 8 probes."""
    rng = np.random.default_rng(seed)
    n = (nx, ny, nz)
    mat = np.zeros((nz, ny, nx), np.uint8)
    table = []
    for b in range(16):
        sl = []
        for a in (2, 1, 0):
            lo, hi = sorted(int(v) for v in rng.integers(0, n[a], 2))
            # a box spans at most half of an axis: about a third of the cells end up dielectric
            sl.append(slice(lo, min(hi + 1, lo + n[a] // 2 + 1)))
        mat[tuple(sl)] = 2 + b
        table.append((float(np.float32(rng.uniform(1.0, 10.0))), float(np.float32(rng.uniform(0.0, 0.05)))))
    c = tuple(v // 2 for v in n)
    mat[c[2] - 2:c[2] + 3, c[1] - 2:c[1] + 3, c[0] - 2:c[0] + 3] = 0  # the port sits in a small air pocket
    w = Workload("hetero", nx, ny, nz, mat.reshape(-1), table, f0=workloads.gaussian_pulse_f0(1e-3), waveform=3,
                 sv=workloads.differentiated_gaussian(steps), steps=steps)
    w.ports.append(([w.cell(*c)], 2, float(np.float32(rng.uniform(0.5, 1.5)))))
    for _ in range(8):  # where the wave arrives early in the run
        w.probes_cell.append(tuple(int(rng.integers(v // 2 - v // 8, v // 2 + v // 8 + 1)) for v in n))
    return w


def _free(nx, ny, nz, steps, seed):
    rng = np.random.default_rng(seed)
    w = Workload("free", nx, ny, nz, np.zeros(nx * ny * nz, np.uint8), [], f0=workloads.gaussian_pulse_f0(1e-3),
                 waveform=2, steps=steps)
    i, j, k = (v // 2 + int(rng.integers(-2, 3)) for v in (nx, ny, nz))
    w.ports.append(([w.cell(i, j, k)], 2, float(np.float32(rng.uniform(0.5, 1.5)))))
    w.probes_cell.append((3 * nx // 4, ny // 2, nz // 2))
    return w


def _dipole(nx, ny, nz, steps, seed):
    w = workloads.random_dipole(np.random.default_rng(seed), nx, ny, nz, steps)
    w.probes_cell.append((3 * nx // 4, ny // 2, nz // 2))
    return w


def _scene(case, seed):
    make = {"hetero": _hetero, "free": _free, "dipole": _dipole}[case["scene"]]
    return make(case["nx"], case["ny"], case["nz"], case["steps"], seed)


def _solve_workload(case, seed):
    w = _scene(case, seed)
    w.rho = case["rho"]
    w.storage = int(STORAGES[case["storage"]])
    w.meta["near_field"] = case["near_field"]
    if w.dft_freqs is None:
        w.dft_freqs = np.linspace(0.5, 1.5, 16) * (w.f0 / 2.0)
    return w


def _mixed(nx, ny, nz, seed):
    """A grid with lossy boxes and scattered PEC cells, and a random state."""
    rng = np.random.default_rng(seed)
    mat = np.zeros((nz, ny, nx), np.uint8)
    mat[nz // 5:nz // 2, ny // 6:ny // 2 + 1, nx // 4:nx - nx // 5] = 2
    mat[nz // 3:nz - 2, ny // 2:, :nx // 2] = 3
    mat[rng.random((nz, ny, nx)) < 0.01] = 1
    v0 = rng.standard_normal((nz, ny, nx, 12), dtype=np.float32)
    v0[mat == 1] = 0.0
    return mat, [(4.5, 0.02), (2.0, 0.0)], v0


def _far_field_workload(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    w = workloads.dipole(nx, ny, nz, max(5, nz // 3), None, steps=case["steps"])
    w.ports[0] = (w.ports[0][0], w.ports[0][1], float(np.float32(rng.uniform(0.5, 1.5))))
    # a carrier that the run resolves over its DFT samples
    w.f0 = float(np.float32(workloads.gaussian_pulse_f0(1e-3, width_steps=rng.uniform(14.0, 18.0))))
    w.meta.update(surface_monitors=True, huy_offset=case["huy"], settle_steps=case["steps"] // 3,
                  field_plane=(1, ny // 2))
    return w


# ---------------------------------------------------------------- the calls

def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return dict(kind=kind, w=_solve_workload(case, seed), state=case.get("state", False))
    if kind == "fdtd":
        return dict(kind=kind, w=_scene(case, seed))
    if kind == "far_field":
        return dict(kind=kind, w=_far_field_workload(case, seed), n=(case["ntheta"], case["nphi"]))
    if kind == "batch":
        return dict(kind=kind, ws=workloads.batched_instances(case["count"], case["steps"], seed=seed, lo=case["lo"],
                                                              hi=case["hi"]))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    mat, table, v0 = _mixed(nx, ny, nz, seed)
    if kind == "resume":
        w = Workload("resume", nx, ny, nz, mat.reshape(-1), table, steps=case["steps"], rho=case["rho"], waveform=3,
                     sv=np.zeros(1, np.float32))
        s = build_solver(w)
        s.stepAsync(0)
        return dict(kind=kind, s=s, v0=v0.reshape(-1), steps=case["steps"])
    # planes: 12 padded pulse planes, 3 stub planes and the tables, on the device
    px = -(-nx // 8) * 8
    dev = torch.device("cuda", torch.cuda.current_device())
    a = torch.zeros((12, nz, ny, px), dtype=torch.float32, device=dev)
    a[..., :nx] = torch.from_numpy(v0).to(dev).permute(3, 0, 1, 2)
    m = torch.ones((nz, ny, px), dtype=torch.uint8, device=dev)
    m[..., :nx] = torch.from_numpy(mat).to(dev)
    y = torch.tensor([4.0 * (e - 1.0) for e, _ in table], dtype=torch.float32, device=dev)
    g = torch.tensor([np.float32(s) * np.float32(1e-3) * np.float32(376.730313) for _, s in table],
                     dtype=torch.float32, device=dev)
    return dict(kind=kind, a=a, b=torch.zeros_like(a), stub=torch.zeros((3, nz, ny, px), device=dev), m=m, y=y, g=g,
                energy=torch.zeros(1, dtype=torch.float64, device=dev), n=(nx, ny, nz), rho=case["rho"],
                lib=_lib.load())


def _records(s, w):
    ports = [s.port(p) for p in range(len(w.ports))]
    probes = [s.probe(q) for q in range(len(w.probes_cell))]
    return ports, probes


def _run_solve(w, state):
    s = build_solver(w)
    s.run()
    ports, probes = _records(s, w)
    v, i = s.portDft(0)
    steps, energy = s.getEnergyHistory(f64=True)
    pulses = s.pulses() if state else np.zeros(0, np.float32)
    s.close()
    return dict(v=ports[0].vRec, i=ports[0].iRec, probes=np.stack([(p.ex, p.ey, p.ez) for p in probes]),
                dft_v=v, dft_i=i, energy_steps=steps, energy=energy, pulses=pulses)


def _run_far_field(w, n):
    s = build_solver(w)
    s.run()
    port = s.port(0)
    js = s.getJsDft()
    huy, _ = s.huygensDft()
    far = s.computeFarField(*n)
    plane, _, _ = s.getFieldPlane()
    s.close()
    return dict(v=port.vRec, i=port.iRec, js=js, huy=huy, U=far["U"], plane=plane)


def _run_batch(ws):
    with Batch() as b:
        got = b.solve(ws, build_solver, lambda s, w: (s.port(0), s.portDft(0)), chunk=32)
    return dict(v=np.stack([p.vRec for p, _ in got]), i=np.stack([p.iRec for p, _ in got]),
                dft_v=np.stack([d[0] for _, d in got]), dft_i=np.stack([d[1] for _, d in got]))


def _run_planes(st):
    nx, ny, nz = st["n"]
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    L = st["lib"]
    status = L.tlm_step_planes_noalloc(p(st["a"]), p(st["b"]), p(st["stub"]), p(st["m"]), p(st["y"]), p(st["g"]),
                                       st["y"].numel(), nx, ny, nz, st["rho"], 0, p(st["energy"]),
                                       C.c_void_p(torch.cuda.current_stream().cuda_stream))
    _lib.check(L, None, status)
    return dict(planes=st["b"], stubs=st["stub"], energy=st["energy"])


def _run_fdtd(w):
    s = build_fdtd(w)
    s.run()
    v, i = s.port(0)
    probes = np.stack([s.probe(q) for q in range(len(w.probes_cell))])
    steps, energy = s.getEnergyHistory(f64=True)
    s.close()
    return dict(v=v, i=i, probes=probes, energy_steps=steps, energy=energy)


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return _run_solve(state["w"], state["state"])
    if kind == "fdtd":
        return _run_fdtd(state["w"])
    if kind == "far_field":
        return _run_far_field(state["w"], state["n"])
    if kind == "batch":
        return _run_batch(state["ws"])
    if kind == "planes":
        return _run_planes(state)
    s = state["s"]
    s.setPulses(state["v0"])
    s.step(state["steps"])
    return dict(pulses=s.pulses(), stubs=s.stubs())


# ------------------------------------------------- what a pass has to move

# additions and multiplications of one node's step: 3 node voltages, 3
# circulations, 12 reflections (TLM); 6 field components (FDTD)
TLM_FLOPS, FDTD_FLOPS = 48, 36


def work(case):
    """A pass reads its inputs once and writes its outputs once: the state
    (12 pulses, or 6 field components, per cell) and the material map. The
    arithmetic is that of every step."""
    kind = case["kind"]
    if kind == "batch":
        cells, steps = case["count"] * ((case["lo"] + case["hi"]) / 2.0) ** 3, case["steps"]
    else:
        cells, steps = case["nx"] * case["ny"] * case["nz"], case.get("steps", 1)
    if kind == "fdtd":
        return {"bytes": cells * (24.0 + 1.0), "flops": float(cells) * steps * FDTD_FLOPS}
    state = 12.0 * BYTES[case.get("storage", "f32")]
    if kind in ("planes", "resume"):
        state *= 2.0
    return {"bytes": cells * (state + 1.0), "flops": float(cells) * steps * TLM_FLOPS}


# ------------------------------------------------- the same in 64 bits

ETA0, C0 = float(np.float32(376.730313)), float(np.float32(299792458.0))
EPS0, MU0 = float(np.float32(8.8541878128e-12)), float(np.float32(1.25663706212e-6))


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _sources(w, dt):
    """Source value of every step."""
    if w.waveform == 3:
        sv = np.zeros(w.steps)
        n = min(w.steps, len(w.sv))
        sv[:n] = w.sv[:n]
        return sv
    tau = 0.5 / w.f0
    u = (np.arange(w.steps) * dt - 3.0 * tau) / tau
    return np.exp(-u * u)


def _first(a):
    return 1 if a == 0 else 0


def _second(a):
    return 1 if a == 2 else 2


def _slot(a, side, f):
    return a * 4 + side * 2 + (0 if f == _first(a) else 1)


def _field(s):
    return _second(s >> 2) if s & 1 else _first(s >> 2)


def _voltage(v, j, at=Ellipsis):
    a, b = (1 if j == 0 else 0), (1 if j == 2 else 2)
    return 0.5 * (v[_slot(a, 0, j)][at] + v[_slot(a, 1, j)][at] + v[_slot(b, 0, j)][at] + v[_slot(b, 1, j)][at])


def _circulation(v, k, at=Ellipsis):
    p, q = (k + 1) % 3, (k + 2) % 3
    return 0.5 * (v[_slot(p, 0, q)][at] - v[_slot(p, 1, q)][at] - v[_slot(q, 0, p)][at] + v[_slot(q, 1, p)][at])


class _Tlm64:
    """The symmetrical condensed node step on 12 incident planes [k, j, i]."""

    def __init__(self, nx, ny, nz, mat, table, dl, rho):
        dev = _dev()
        self.n, self.rho, self.dl = (nx, ny, nz), rho, dl
        m = torch.from_numpy(np.ascontiguousarray(mat).reshape(nz, ny, nx)).to(dev)
        self.v = [torch.zeros((nz, ny, nx), dtype=torch.float64, device=dev) for _ in range(12)]
        pec = m == 1
        self.pec = pec.reshape(-1).nonzero().reshape(-1)
        self.pec_next = {}
        for a in range(3):
            for side in (0, 1):
                near = torch.zeros_like(pec)
                dst, src = self._shift(a, side)
                near[dst] = pec[src]
                self.pec_next[a, side] = near.reshape(-1).nonzero().reshape(-1)
        self.diel = (m >= 2).reshape(-1).nonzero().reshape(-1)
        if len(self.diel):
            yh = torch.tensor([4.0 * (max(1.0, float(np.float32(e))) - 1.0) for e, _ in table], dtype=torch.float64)
            gh = torch.tensor([max(0.0, float(np.float32(s))) * float(np.float32(dl)) * ETA0 for _, s in table],
                              dtype=torch.float64)
            ids = m.reshape(-1)[self.diel].long() - 2
            self.yh, self.gh = yh.to(dev)[ids], gh.to(dev)[ids]
            self.vs = [torch.zeros(len(self.diel), dtype=torch.float64, device=dev) for _ in range(3)]

    def _shift(self, a, side):
        """Cells with a neighbour on that side along axis a, and those neighbours."""
        dst, src = [slice(None)] * 3, [slice(None)] * 3
        dst[2 - a], src[2 - a] = (slice(0, -1), slice(1, None)) if side else (slice(1, None), slice(0, -1))
        return tuple(dst), tuple(src)

    def scatter(self):
        v, out = self.v, []
        V = [_voltage(v, j) for j in range(3)]
        if len(self.diel):
            for j in range(3):
                flat = V[j].reshape(-1)
                num = 2.0 * (2.0 * flat[self.diel] + self.yh * self.vs[j])
                vj = num / (4.0 + self.yh + self.gh)
                flat[self.diel] = vj
                self.vs[j] = vj - self.vs[j]
        Z = [_circulation(v, k) for k in range(3)]
        for s in range(12):
            i, side, j = s >> 2, (s >> 1) & 1, _field(s)
            sign = 1.0 if (j == (i + 1) % 3) == (side == 1) else -1.0
            r = V[j] + sign * Z[3 - i - j] - v[s ^ 2]
            if len(self.pec):
                r.reshape(-1)[self.pec] = 0.0
            out.append(r)
        self.v = out

    def connect(self):
        r, inc = self.v, []
        for s in range(12):
            a, side = s >> 2, (s >> 1) & 1
            x = torch.empty_like(r[s])
            dst, src = self._shift(a, side)
            x[dst] = r[s ^ 2][src]
            wall = [slice(None)] * 3
            wall[2 - a] = -1 if side else 0
            x[tuple(wall)] = self.rho * r[s][tuple(wall)]
            near = self.pec_next[a, side]
            if len(near):
                x.reshape(-1)[near] = -r[s].reshape(-1)[near]
            if len(self.pec):
                x.reshape(-1)[self.pec] = 0.0
            inc.append(x)
        self.v = inc

    def inject(self, cell, pol, q):
        for s in range(12):
            if (s >> 2) != pol and _field(s) == pol:
                self.v[s].view(-1)[cell] += q

    def energy(self):
        return sum((x * x).sum() for x in self.v)


def _tlm64(w, monitor=None):
    """Records of a workload's solve: v, i, probes, energy steps and energy."""
    t = _Tlm64(w.nx, w.ny, w.nz, w.mat, w.table, w.dl, w.rho)
    dl = float(np.float32(w.dl))
    dt = dl / (2.0 * C0)
    sv = _sources(w, dt)
    cells, pol, amp = w.ports[0]
    cells = [int(c) for c in cells if w.mat[int(c)] == 0]
    stride = (1, w.nx, w.nx * w.ny)
    mid = cells[len(cells) // 2]
    t1, t2 = (pol + 1) % 3, (pol + 2) % 3
    loop = [mid + stride[t1], mid - stride[t1], mid + stride[t2], mid - stride[t2]]
    probe = [w.cell(*c) for c in w.probes_cell]
    at = torch.tensor(cells + loop + probe, device=_dev())
    smp, energy = [], []
    for n in range(w.steps):
        for c in cells:
            t.inject(c, pol, 0.5 * amp * float(sv[n]))
        if monitor is not None:
            monitor(n, t, dt)
        s = [x.reshape(-1)[at] for x in t.v]
        smp.append(torch.stack([_voltage(s, j) for j in range(3)] + [_circulation(s, k) for k in range(3)]))
        if n % 16 == 0:
            energy.append(t.energy())
        t.scatter()
        t.connect()
    smp = torch.stack(smp).cpu().numpy()          # [step, 6, point]
    nc = len(cells)
    v = smp[:, pol, :nc].sum(1)
    zi = smp[:, 3 + t2, nc] - smp[:, 3 + t2, nc + 1] - smp[:, 3 + t1, nc + 2] + smp[:, 3 + t1, nc + 3]
    return dict(v=v, i=-2.0 * zi / ETA0, probes=(-smp[:, :3, nc + 4:] / dl).transpose(2, 1, 0),
                energy_steps=None, energy=torch.stack(energy).cpu().numpy(), dt=dt, t=t)


def _dft(x, freqs, dt):
    ph = np.outer(2.0 * np.pi * np.asarray(freqs) * dt, np.arange(len(x)))
    return (np.cos(ph) - 1j * np.sin(ph)) @ x


def _exact_solve(w, state=False):
    r = _tlm64(w)
    dt, t = r.pop("dt"), r.pop("t")
    pulses = torch.stack(t.v).permute(1, 2, 3, 0).reshape(-1) if state else np.zeros(0)
    return dict(r, pulses=pulses, dft_v=_dft(r["v"], w.dft_freqs, dt), dft_i=_dft(r["i"], w.dft_freqs, dt))


def _pec_faces(w):
    """(cell next to a PEC cell, axis) in cell, axis, side order."""
    m = w.mat.reshape(w.nz, w.ny, w.nx)
    out = []
    for k, j, i in np.argwhere(m == 1):
        for a in range(3):
            for sd in (-1, 1):
                c = [i, j, k]
                c[a] += sd
                if 0 <= c[a] < (w.nx, w.ny, w.nz)[a] and m[c[2], c[1], c[0]] != 1:
                    out.append((w.cell(*c), a))
    return out


def _huygens_faces(w, o):
    """(cell, axis, outward sign, position from the grid centre)."""
    n = (w.nx, w.ny, w.nz)
    lo, hi = (o, o, o), tuple(v - 1 - o for v in n)
    out = []
    for a, slow, fast in ((0, 2, 1), (1, 2, 0), (2, 1, 0)):
        for p in range(lo[slow], hi[slow] + 1):
            for q in range(lo[fast], hi[fast] + 1):
                for sign in (-1, 1):
                    c = [0, 0, 0]
                    c[slow], c[fast], c[a] = p, q, (lo[a] if sign < 0 else hi[a])
                    if w.mat[w.cell(*c)] == 0:
                        out.append((w.cell(*c), a, sign, [(c[x] + 0.5) * w.dl - 0.5 * n[x] * w.dl for x in range(3)]))
    return out


def _exact_far_field(w, ntheta, nphi):
    dev = _dev()
    faces, huy = _pec_faces(w), _huygens_faces(w, w.meta["huy_offset"])
    axis_f = torch.tensor([a for _, a in faces], device=dev)
    at_f = torch.tensor([c for c, _ in faces], device=dev)
    axis_h = torch.tensor([f[1] for f in huy], device=dev)
    at_h = torch.tensor([f[0] for f in huy], device=dev)
    first, second = torch.tensor([1, 0, 0], device=dev), torch.tensor([2, 2, 1], device=dev)
    js = torch.zeros((len(faces), 4), dtype=torch.float64, device=dev)
    acc = torch.zeros((len(huy), 8), dtype=torch.float64, device=dev)
    last = {}
    f0 = float(np.float32(w.f0))

    def tangential(t, at, axis, of):
        s = [x.reshape(-1)[at] for x in t.v]
        q = torch.stack([of(s, j) for j in range(3)])
        r = torch.arange(len(at), device=dev)
        return q[first[axis], r], q[second[axis], r]

    def monitor(n, t, dt):
        if n % 2 == 0:
            j = w.meta["field_plane"][1]
            last["plane"] = sum(_voltage(t.v, q, (slice(None), j)) ** 2 for q in range(3)).sqrt()
        if n < w.meta["settle_steps"]:
            return
        c, s = math.cos(2.0 * math.pi * f0 * n * dt), math.sin(2.0 * math.pi * f0 * n * dt)
        last["samples"] = last.get("samples", 0) + 1
        h1, h2 = tangential(t, at_f, axis_f, _circulation)
        js.add_(torch.stack([h1 * c, -h1 * s, h2 * c, -h2 * s], 1))
        e1, e2 = tangential(t, at_h, axis_h, _voltage)
        m1, m2 = tangential(t, at_h, axis_h, _circulation)
        acc.sub_(torch.stack([e1 * c, -e1 * s, e2 * c, -e2 * s, m1 * c, -m1 * s, m2 * c, -m2 * s], 1))

    r = _tlm64(w, monitor)
    # the magnitude of a face's DFT, normalised by the samples taken
    mag = (2.0 / max(1, last["samples"])) * js.square().sum(1).sqrt()
    # equivalent currents on the box, and their radiation vectors
    sa = torch.where(axis_h == 1, -1.0, 1.0).double() * torch.tensor([float(f[2]) for f in huy], device=dev).double()
    e1, e2 = torch.complex(acc[:, 0], acc[:, 1]), torch.complex(acc[:, 2], acc[:, 3])
    m1, m2 = torch.complex(acc[:, 4], acc[:, 5]), torch.complex(acc[:, 6], acc[:, 7])
    row = torch.arange(len(huy), device=dev)
    J = torch.zeros((3, len(huy)), dtype=torch.complex128, device=dev)
    M = torch.zeros_like(J)
    J[second[axis_h], row], J[first[axis_h], row] = sa * m1, -sa * m2
    M[second[axis_h], row], M[first[axis_h], row] = -sa * e1, sa * e2
    pos = torch.tensor([f[3] for f in huy], dtype=torch.float64, device=dev)
    k0 = 2.0 * math.pi * f0 / C0
    U = np.zeros((ntheta, nphi))
    for a in range(ntheta):
        th = math.pi * a / (ntheta - 1)
        ph = 2.0 * math.pi * torch.arange(nphi, dtype=torch.float64, device=dev) / (nphi - 1)
        cp, sp, st, ct = ph.cos(), ph.sin(), math.sin(th), math.cos(th)
        z = torch.zeros_like(cp)
        rh, tv, pv = (torch.stack(x) for x in ((st * cp, st * sp, z + ct), (ct * cp, ct * sp, z - st), (-sp, cp, z)))
        wave = torch.exp(1j * k0 * (pos @ rh))
        N, L = J @ wave, M @ wave
        Nt, Np, Lt, Lp = (N * tv).sum(0), (N * pv).sum(0), (L * tv).sum(0), (L * pv).sum(0)
        U[a] = ((Lp + Nt).abs() ** 2 + (Lt - Np).abs() ** 2).cpu().numpy()
    return dict(v=r["v"], i=r["i"], js=mag.cpu().numpy(), huy=acc.cpu().numpy(), U=U,
                plane=last["plane"].cpu().numpy())


def _exact_mixed(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    mat, table, v0 = _mixed(nx, ny, nz, seed)
    t = _Tlm64(nx, ny, nz, mat, table, 1e-3, case["rho"])
    t.v = [torch.from_numpy(np.ascontiguousarray(v0[..., s])).to(_dev()).double() for s in range(12)]
    planes = case["kind"] == "planes"
    energy = None
    if planes:  # the input planes hold reflected pulses
        t.connect()
        energy = t.energy().reshape(1)
    for _ in range(1 if planes else case["steps"]):
        t.scatter()
        if not planes:
            t.connect()
    vs = torch.zeros((3, nx * ny * nz), dtype=torch.float64, device=_dev())
    for j in range(3):
        vs[j, t.diel] = t.vs[j]
    v = torch.stack(t.v)
    if not planes:
        return dict(pulses=v.permute(1, 2, 3, 0).reshape(-1), stubs=vs.t().reshape(-1))
    pad = (0, -nx % 8)
    return dict(planes=torch.nn.functional.pad(v, pad),
                stubs=torch.nn.functional.pad(vs.reshape(3, nz, ny, nx), pad), energy=energy)


def _fdtd_coefficients(w, dt, axis, ext):
    """PEC mask and (ca, cb) of every E edge along `axis`, [k, j, i]."""
    dev = _dev()
    m = torch.from_numpy(w.mat.reshape(w.nz, w.ny, w.nx)).to(dev).long()
    er = torch.tensor([1.0, 1.0] + [float(np.float32(e)) for e, _ in w.table], dtype=torch.float64, device=dev)[m]
    sg = torch.tensor([0.0, 0.0] + [float(np.float32(s)) for _, s in w.table], dtype=torch.float64, device=dev)[m]
    shape = tuple(reversed(ext))
    acc = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(4)]
    t1, t2 = 2 - _first(axis), 2 - _second(axis)
    for d1 in (0, 1):
        for d2 in (0, 1):
            sl = [slice(None)] * 3
            sl[t1], sl[t2] = slice(d1, d1 + m.shape[t1]), slice(d2, d2 + m.shape[t2])
            for a, x in zip(acc, (er, sg, torch.ones_like(er), (m == 1).double())):
                a[tuple(sl)] += x
    eps = EPS0 * torch.clamp(acc[0] / acc[2], min=1.0)
    lf = (acc[1] / acc[2]) * dt / (2.0 * eps)
    free = acc[3] == 0
    return ((1.0 - lf) / (1.0 + lf)) * free, (dt / (eps * float(np.float32(w.dl)))) / (1.0 + lf) * free


def _exact_fdtd(w):
    dev = _dev()
    nx, ny, nz = w.nx, w.ny, w.nz
    dl = float(np.float32(w.dl))
    dt = float(np.float32(0.99)) * dl / (C0 * math.sqrt(3.0))
    ch, mur = dt / (MU0 * dl), (C0 * dt - dl) / (C0 * dt + dl)
    eext = ((nx, ny + 1, nz + 1), (nx + 1, ny, nz + 1), (nx + 1, ny + 1, nz))
    hext = ((nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1))
    zeros = lambda e: torch.zeros(tuple(reversed(e)), dtype=torch.float64, device=dev)  # noqa: E731
    E, H = [zeros(e) for e in eext], [zeros(e) for e in hext]
    co = [_fdtd_coefficients(w, dt, a, eext[a]) for a in range(3)]
    sv = _sources(w, dt)
    cells, pol, amp = w.ports[0]
    cells = [int(c) for c in cells if w.mat[int(c)] == 0]
    ijk = lambda c: (c % nx, (c // nx) % ny, c // (nx * ny))  # noqa: E731

    def around(c, pol):
        """The four E edges of a cell along pol, as [k, j, i]."""
        out = []
        for d1 in (0, 1):
            for d2 in (0, 1):
                q = list(c)
                q[_first(pol)] += d2
                q[_second(pol)] += d1
                out.append((q[2], q[1], q[0]))
        return out

    def ec(c, a):
        return 0.25 * sum(E[a][q] for q in around(c, a))

    def hc(c, a):
        q = list(c)
        q[a] += 1
        return 0.5 * (H[a][c[2], c[1], c[0]] + H[a][q[2], q[1], q[0]])

    def off(c, a, d):
        q = list(c)
        q[a] += d
        return tuple(q)

    def diff(x, a):
        d = 2 - a
        return x.narrow(d, 1, x.shape[d] - 1) - x.narrow(d, 0, x.shape[d] - 1)

    t1, t2 = (pol + 1) % 3, (pol + 2) % 3
    mid = ijk(cells[len(cells) // 2])
    v, cur, probes, energy = [], [], [], []
    for n in range(w.steps):
        for c in cells:
            for q in around(ijk(c), pol):
                if co[pol][1][q] != 0.0:
                    E[pol][q] += -0.25 * amp * float(sv[n])
        v.append(-dl * sum(ec(ijk(c), pol) for c in cells))
        cur.append(2.0 * dl * (hc(off(mid, t1, 1), t2) - hc(off(mid, t1, -1), t2)
                               - hc(off(mid, t2, 1), t1) + hc(off(mid, t2, -1), t1)))
        probes.append(torch.stack([torch.stack([ec(c, a) for a in range(3)]) for c in w.probes_cell]))
        if n % 16 == 0:
            energy.append(sum((x * x).sum() for x in E) + ETA0 * ETA0 * sum((x * x).sum() for x in H))
        for a in range(3):
            p, q = (a + 1) % 3, (a + 2) % 3
            H[a] = H[a] - ch * (diff(E[q], p) - diff(E[p], q))
        old = [x.clone() for x in E]
        for a in range(3):
            p, q = (a + 1) % 3, (a + 2) % 3
            dp, dq = 2 - p, 2 - q
            curl = diff(H[q], p).narrow(dq, 1, H[q].shape[dq] - 2) - diff(H[p], q).narrow(dp, 1, H[p].shape[dp] - 2)
            sl = [slice(None)] * 3
            sl[dp], sl[dq] = slice(1, -1), slice(1, -1)
            sl = tuple(sl)
            E[a][sl] = co[a][0][sl] * E[a][sl] + co[a][1][sl] * curl
        for face in range(3):
            for a in range(3):
                if a == face:
                    continue
                d = 2 - face
                for b, i in ((0, 1), (E[a].shape[d] - 1, E[a].shape[d] - 2)):
                    E[a].select(d, b).copy_(old[a].select(d, i)
                                            + mur * (E[a].select(d, i) - old[a].select(d, b)))
    return dict(v=torch.stack(v).cpu().numpy(), i=torch.stack(cur).cpu().numpy(),
                probes=torch.stack(probes, -1).cpu().numpy(), energy_steps=None,
                energy=torch.stack(energy).cpu().numpy())


def exact(case, seed):
    kind = case["kind"]
    cells = case.get("nx", 0) * case.get("ny", 0) * case.get("nz", 0)
    # a step in 64 bits launches some hundred kernels and moves about 2 kB a cell
    count = case["count"] if kind == "batch" else 1
    if kind == "batch":
        cells = ((case["lo"] + case["hi"]) / 2.0) ** 3
    if case.get("steps", 1) * count * (1.5e-3 + cells * 1.2e-9) > 20.0:
        return None
    if kind == "solve":
        return _exact_solve(_solve_workload(case, seed), case.get("state", False))
    if kind == "fdtd":
        return _exact_fdtd(_scene(case, seed))
    if kind == "far_field":
        return _exact_far_field(_far_field_workload(case, seed), case["ntheta"], case["nphi"])
    if kind == "batch":
        got = []
        for w in workloads.batched_instances(case["count"], case["steps"], seed=seed, lo=case["lo"], hi=case["hi"]):
            got.append(_exact_solve(w))
        return {k: np.stack([r[k] for r in got]) for k in ("v", "i", "dft_v", "dft_i")}
    return _exact_mixed(case, seed)
