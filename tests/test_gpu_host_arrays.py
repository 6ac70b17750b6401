"""State transfers of small systems from and to every kind of host array: pageable, pinned,
pinned with an offset, registered by its owner, and pinned but off the 8-byte boundary
that the GPU needs to reach into it by itself."""

import ctypes

import numpy as np
import pytest

import ljref

pytestmark = pytest.mark.gpu

N = 2000


class Host:
    """An N x 4 array of doubles in host memory of some kind."""

    def __init__(self, kind):
        import torch
        self.rt, self.registered = torch.cuda.cudart(), None
        size = N * 32
        if kind in ("pinned", "offset", "odd"):
            self.hold = torch.empty(size + 64, dtype=torch.uint8, pin_memory=True)
            at = {"pinned": 0, "offset": 8, "odd": 4}[kind]
            buf = self.hold.numpy()
        else:
            buf = self.hold = np.zeros(size + 16384, dtype=np.uint8)[4096:]
            at = 0
            if kind == "registered":  # ends at a page's end
                at = -(buf.ctypes.data + size) % 4096
                start = (buf.ctypes.data + at) // 4096 * 4096
                self.registered = start
                assert int(self.rt.cudaHostRegister(start, buf.ctypes.data + at + size - start, 0)) == 0
        self.a = np.ndarray((N, 4), np.float64, buf.data, at)
        self.p = ctypes.c_void_p(self.a.__array_interface__["data"][0])

    def close(self):
        if self.registered:
            assert int(self.rt.cudaHostUnregister(self.registered)) == 0


@pytest.mark.parametrize("kind", ["pageable", "pinned", "offset", "odd", "registered"])
@pytest.mark.parametrize("batch", [False, True])
def test_transfers(kind, batch):
    import torch
    from lennardjonesium import GpuSystem
    from lennardjonesium import _native as nat
    torch.zeros(1, device="cuda")
    x, v, L = ljref.initial_state(N, 1.0, 0.8, 4)
    a, b, c = Host(kind), Host(kind), Host(kind)
    lib, h = nat.lib(), ctypes.c_void_p()
    try:
        a.a[:], b.a[:] = x, v
        if batch:
            table = (nat.BatchSystem * 1)()
            table[0].particle_count, table[0].time_delta, table[0].skin = N, 0.005, -1.0
            for k in range(3):
                table[0].box[k] = L
            nat.check(lib.lj_batch_create(table, 1, 2.5, 0, ctypes.byref(h)))
            assert lib.lj_batch_upload_system(h, 0, a.p, b.p, 4) == 0
            assert lib.lj_batch_step(h, 3, None) == 0
            a.a[:], b.a[:], c.a[:] = -1.0, -1.0, -1.0
            assert lib.lj_batch_download_system(h, 0, a.p, b.p, c.p, 4) == 0
        else:
            g = GpuSystem(N, L)
            assert lib.lj_gpu_upload_state(g._ctx, a.p, b.p, None, None, 4, 0.0, 0.0, 0.0) == 0
            g.step(3)
            a.a[:], b.a[:], c.a[:] = -1.0, -1.0, -1.0
            assert lib.lj_gpu_download_state(g._ctx, a.p, b.p, None, c.p, 4, None, None, None) == 0
            g.close()
        with GpuSystem(N, L) as g:
            g.upload(x, v=v)
            g.step(3)
            want = g.download()
        for got, k in ((a, "x"), (b, "v"), (c, "F")):
            assert np.array_equal(got.a[:, :3], want[k][:, :3]), k
    finally:
        if h:
            lib.lj_batch_destroy(h)
        for q in (a, b, c):
            q.close()
