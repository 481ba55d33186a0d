"""Energies of the allocation-free step after calls that shared a scratch slot.

Replays of two captured calls on one slot, of different sizes, overlap on two
streams: their own energies are undefined by the contract, but every call after
them, on any slot, and every replay that runs alone give the energy of their
own input, bitwise that of the same call before."""
import ctypes as C

import pytest

from emsolver_b200 import _lib

pytestmark = pytest.mark.gpu

SLOTS = 16


def test_collisions_harm_no_later_call(built):
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda", 0)
    L = _lib.load()

    class Planes:
        def __init__(self, n, seed):
            self.n = n
            g = torch.Generator(device=dev).manual_seed(seed)
            self.a = torch.randn(12 * n ** 3, device=dev, generator=g)
            self.b = torch.empty_like(self.a)
            self.mat = torch.zeros(n ** 3, dtype=torch.uint8, device=dev)
            self.e = torch.full((1,), float("nan"), dtype=torch.float64, device=dev)

        def call(self):
            st = L.tlm_step_planes_noalloc(self.a.data_ptr(), self.b.data_ptr(), None, self.mat.data_ptr(), None, None,
                                           0, self.n, self.n, self.n, 0.0, 0, self.e.data_ptr(),
                                           C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
            assert st == _lib.TLM_OK, L.tlm_last_error(None)

        def energy(self, run):
            self.e.fill_(float("nan"))
            torch.cuda.synchronize(dev)
            run()
            torch.cuda.synchronize(dev)
            return self.e.item()

    big, small, other = Planes(160, 1), Planes(24, 2), Planes(40, 3)
    want = [p.energy(p.call) for p in (big, small, other)]
    assert all(w > 0.0 for w in want)

    def capture(p):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            p.call()
        return g

    graphs = [capture(big)]
    for _ in range(SLOTS - 1):
        other.call()
    graphs.append(capture(small))     # the same slot
    streams = [torch.cuda.Stream(dev) for _ in range(2)]
    for _ in range(60):
        with torch.cuda.stream(streams[0]):
            graphs[0].replay()
        for _ in range(8):
            with torch.cuda.stream(streams[1]):
                graphs[1].replay()
    torch.cuda.synchronize(dev)
    for _ in range(2 * SLOTS):
        assert other.energy(other.call) == want[2]
    assert big.energy(graphs[0].replay) == want[0]
    assert small.energy(graphs[1].replay) == want[1]
    assert small.energy(graphs[1].replay) == want[1]
    for _ in range(2 * SLOTS):
        assert other.energy(other.call) == want[2]
