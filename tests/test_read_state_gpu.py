"""The state on the host: five arrays of the caller's own, also page-locked
ones that happen to lie next to each other, and one array for all planes."""
import ctypes as C
import mmap

import numpy as np
import pytest

from helpers import small

pytestmark = pytest.mark.gpu

from fvm_b200 import Batch, Server, Solver, abi  # noqa: E402

torch = pytest.importorskip("torch")

# planes of whole pages; the second one's rows are narrower than the device's
GRIDS = [(64, 64), (48, 64)]


class Adjacent:
    """Five page-locked arrays, each registered on its own, one behind the other."""

    def __init__(self, nx, ny):
        self.bytes = nx * ny * 4
        assert self.bytes % mmap.PAGESIZE == 0
        self.array = np.frombuffer(mmap.mmap(-1, 5 * self.bytes), np.float32).reshape(5, ny, nx)
        self.ptrs = [self.array.ctypes.data + k * self.bytes for k in range(5)]

    def __enter__(self):
        for p in self.ptrs:
            assert int(torch.cuda.cudart().cudaHostRegister(p, self.bytes, 0)) == 0
        return self

    def __exit__(self, *exc):
        for p in self.ptrs:
            assert int(torch.cuda.cudart().cudaHostUnregister(p)) == 0


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("nx,ny", GRIDS)
def test_read_fields_into_arrays_of_the_caller_s_own(nx, ny):
    p, e = small("euler_m3_circle", nx, ny)
    s = Solver(p, e)
    p.dt = 0.5 * s.compute_dt()
    s.step(3)
    ref = s.fields()
    assert _same(ref, s.read_region(0, 0, nx, ny))
    with Adjacent(nx, ny) as a:
        assert s.lib.fvm_read_fields(s.h, *[C.c_void_p(p) for p in a.ptrs]) == 0
        assert _same(a.array, ref)
    one = np.zeros((ny, nx), np.float32)
    assert s.lib.fvm_read_fields(s.h, None, None, C.c_void_p(one.ctypes.data), None, None) == 0
    assert _same(one, ref[2])
    assert s.lib.fvm_read_state(s.h, None) == 1


@pytest.mark.parametrize("nx,ny", GRIDS)
def test_batch_and_server_states(nx, ny):
    p, e = small("euler_m3_circle", nx, ny)
    e.dt_policy = abi.DT_RECOMPUTE
    b = Batch(e)
    i = b.add(p)
    b.step(5)
    ref = b.fields(i)
    q, _ = small("euler_m3_circle", nx, ny)
    s = Solver(q, e)
    s.step(5)
    assert _same(ref, s.fields())
    with Adjacent(nx, ny) as a:
        assert b.lib.fvm_batch_read_fields(b.h, i, *[C.c_void_p(p) for p in a.ptrs]) == 0
        assert _same(a.array, ref)
    assert b.lib.fvm_batch_read_state(b.h, i, None) == 1
    srv = Server(e, budget_bytes=10**9)
    try:
        r, got = srv.wait(srv.submit(p, 5))
        assert r.status == 0 and _same(got, ref)
        r, got = srv.wait(srv.submit(p, 5, keep_fields=False))
        assert r.status == 0 and got is None
        with Adjacent(nx, ny) as a:
            t = C.c_longlong()
            assert srv.lib.fvm_server_submit(srv.h, C.byref(p), 5, *[C.c_void_p(x) for x in a.ptrs], C.byref(t)) == 0
            assert srv.wait(t.value)[0].status == 0
            assert _same(a.array, ref)
    finally:
        srv.close()
