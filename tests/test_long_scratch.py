"""swift_sw_pairs' direction scratch for long pairs where memory is short: the
rounded size, the second region and the packed launches' regions are given up
before a call fails.  The device's memory pool is replaced by one of a fixed
largest size; results are compared with a call that had all it asked for."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LONG_BYTES = 256 * 4 * (8256 + 32)  # direction words of a pair with an 8,192-base window


class PoolProps(C.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("loc_type", C.c_int),
                ("loc_id", C.c_int), ("security", C.c_void_p), ("max_size", C.c_size_t),
                ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


class CappedPool:
    def __init__(self, size):
        self.cu = C.CDLL("libcuda.so.1")
        self.pool, props = C.c_void_p(), PoolProps(alloc_type=1, loc_type=1, max_size=size)
        assert self.cu.cuMemPoolCreate(C.byref(self.pool), C.byref(props)) == 0

    def __enter__(self):
        assert self.cu.cuDeviceSetMemPool(0, self.pool) == 0

    def __exit__(self, *a):
        default = C.c_void_p()
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(default), 0) == 0
        assert self.cu.cuDeviceSetMemPool(0, default) == 0
        assert self.cu.cuMemPoolDestroy(self.pool) == 0


@pytest.mark.parametrize("n_long,packed,cap", [
    # one region: exact it fits, rounded to whole GiB it does not
    (140, (), 1.6),
    # two launches of 8 GB each: one region fits
    (1000, (), 10),
    # exact it fits once the two regions of the packed launches are back
    (140, ((100, 500, 30_000), (128, 500, 30_000)), 1.6),
])
def test_scratch_that_memory_allows(n_long, packed, cap):
    from swift_gb300 import build as b
    b.build()
    import swift_gb300 as sg
    rng = np.random.default_rng(n_long + len(packed))
    ref = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 1_000_000)].tobytes()
    ql = np.concatenate([np.full(n_long, 300)] + [np.full(n, q) for q, _, n in packed])
    rl = np.concatenate([np.full(n_long, 8192)] + [np.full(n, r) for _, r, n in packed])
    ro = rng.integers(0, len(ref) - 8192, len(ql))
    qo = ro + rng.integers(0, rl - ql)
    need = n_long * LONG_BYTES
    assert need > 1 << 30 and (n_long > 942 or need < cap * 2**30)
    args = (ref, qo, ql, ref, ro, rl)

    def call():
        ctx = sg.Context(0)
        try:
            return ctx.sw_pairs(*args, consensus=False)[0]
        finally:
            ctx.close()

    want = call()
    assert (want["score"] == 2 * ql).all()
    with CappedPool(int(cap * 2**30)):
        got = call()
    for k in ("score", "start", "end", "len"):
        assert np.array_equal(got[k], want[k]), k
