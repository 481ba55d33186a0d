"""The far field against its FP64 evaluation from the same Huygens phasors.

Direction counts that leave the last group of four ragged, face lists in one
slice and in several. Bound: a face's phase k0 r.pos is a few FP32 operations on
terms of size k0 |r||pos|, the sine and cosine are within two units of
the last place and the unit vectors within a few, so the sums N and L are off by
at most delta = 2^-23 (6 + 2 max phase) A, A the sum of the faces' current
magnitudes, and U = |.|^2 + |.|^2 by 2 sqrt(2 U) * 2 delta + 8 delta^2. The sums
themselves are FP64; U is returned in FP32."""
import numpy as np
import pytest

from emsolver_b200 import workloads
from emsolver_b200.runner import build_solver

pytestmark = pytest.mark.gpu


def reference(s, w, nt, npk):
    f, acc = s.huygensFaces(), s.huygensDft()[0].astype(np.float64)
    ax, sg = f["axis"], f["out_sign"].astype(np.float64)
    n = len(ax)
    sa = np.where(ax == 1, -1.0, 1.0) * sg
    t1, t2 = np.where(ax == 0, 1, 0), np.where(ax == 2, 1, 2)
    e1, e2, m1, m2 = (acc[:, 2 * q] + 1j * acc[:, 2 * q + 1] for q in range(4))
    J, M = np.zeros((3, n), complex), np.zeros((3, n), complex)
    r = np.arange(n)
    J[t2, r], J[t1, r], M[t2, r], M[t1, r] = sa * m1, -sa * m2, -sa * e1, sa * e2
    k0 = 2 * np.pi * float(np.float32(w.f0)) / 299792458.0
    pos = f["pos"].astype(np.float64)
    U = np.zeros((nt, npk))
    for i in range(nt):
        for j in range(npk):
            th, ph = np.pi * i / (nt - 1), 2 * np.pi * j / (npk - 1)
            rh = np.array([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)])
            tv = np.array([np.cos(th) * np.cos(ph), np.cos(th) * np.sin(ph), -np.sin(th)])
            pv = np.array([-np.sin(ph), np.cos(ph), 0.0])
            e = np.exp(1j * k0 * (pos @ rh))
            N, L = J @ e, M @ e
            U[i, j] = abs(L @ pv + N @ tv) ** 2 + abs(L @ tv - N @ pv) ** 2
    A = np.abs(J).sum() + np.abs(M).sum()
    delta = 2.0 ** -23 * (6 + 2 * k0 * np.linalg.norm(pos, axis=1).max()) * A
    return U, 2 * np.sqrt(2 * U) * 2 * delta + 8 * delta ** 2 + 2.0 ** -23 * U


@pytest.mark.parametrize("size,directions", [((17, 14, 16), (2, 3)), ((17, 14, 16), (5, 9)), ((50, 46, 53), (3, 3)),
                                             ((50, 46, 53), (13, 25)), ((64, 61, 70), (19, 37))])
def test_far_field_against_fp64(built, size, directions):
    nx, ny, nz = size
    w = workloads.dipole(nx, ny, nz, max(3, nz // 3), None, steps=60)
    w.f0 = float(np.float32(workloads.gaussian_pulse_f0(1e-3, width_steps=15.0)))
    w.meta.update(surface_monitors=True, huy_offset=2, settle_steps=5)
    s = build_solver(w)
    s.step(w.steps)
    U = s.computeFarField(*directions)["U"].astype(np.float64)
    ref, bound = reference(s, w, *directions)
    assert ref.max() > 0 and np.all(np.abs(U - ref) <= bound)
