"""Device blocks take the memory that was asked for, to cudaMalloc's granularity."""
import ctypes as C

import pytest
import torch

from jfem_b200 import _native as N

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("size", [1 << 20, 33 * MB + 1, 100 * MB + 1, 250 * MB + 1, 256 * MB, 256 * MB + 1, 273 * MB + 1,
                                  1100 * MB + 1])
def test_block_size(size):
    lib = N.load()
    alloc, free = lib["_ZN3jfg10pool_allocEmPi"], lib["_ZN3jfg9pool_freeEPvmi"]
    alloc.restype, alloc.argtypes = C.c_void_p, [C.c_size_t, C.POINTER(C.c_int)]
    free.restype, free.argtypes = None, [C.c_void_p, C.c_size_t, C.c_int]
    ctx = N.Context(0)
    ctx.check(lib.jfg_release_scratch(ctx.handle))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    dev = C.c_int(-1)
    p = alloc(size, C.byref(dev))
    used = before - torch.cuda.mem_get_info()[0]
    free(p, size, dev.value)
    ctx.check(lib.jfg_release_scratch(ctx.handle))
    assert dev.value == 0 and torch.cuda.mem_get_info()[0] == before
    # the driver takes multiples of 2 MB
    assert used <= size + 4 * MB, (size, used)
