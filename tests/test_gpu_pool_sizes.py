"""Device blocks take the memory that was asked for, to cudaMalloc's granularity."""
import ctypes as C

import pytest
import torch

from jfem_b200 import _native as N

pytestmark = pytest.mark.gpu

MB = 1 << 20


def pool(lib):
    alloc, free = lib["_ZN3jfg10pool_allocEmPi"], lib["_ZN3jfg9pool_freeEPvmi"]
    alloc.restype, alloc.argtypes = C.c_void_p, [C.c_size_t, C.POINTER(C.c_int)]
    free.restype, free.argtypes = None, [C.c_void_p, C.c_size_t, C.c_int]
    return lambda size: alloc(size, C.byref(C.c_int(-1))), lambda p, size: free(p, size, 0)


def test_a_full_pool_keeps_what_was_released_last():
    alloc, free = pool(N.load())
    ctx = N.Context(0)
    ctx.check(N.load().jfg_release_scratch(ctx.handle))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    first = [alloc(64 * MB) for _ in range(20)]      # more than the pool keeps, of one size
    for p in first:
        free(p, 64 * MB)
    kept = before - torch.cuda.mem_get_info()[0]
    assert 1000 * MB <= kept <= 1024 * MB + 4 * MB
    p = alloc(33 * MB)                               # another size, again and again
    for _ in range(3):
        free(p, 33 * MB)
        held = torch.cuda.mem_get_info()[0]
        assert before - held <= 1024 * MB + 4 * MB
        assert alloc(33 * MB) == p and torch.cuda.mem_get_info()[0] == held
    free(p, 33 * MB)
    newest = alloc(64 * MB)
    assert newest == first[-1]                       # of a size the newest, the oldest are gone
    free(newest, 64 * MB)
    ctx.check(N.load().jfg_release_scratch(ctx.handle))
    assert torch.cuda.mem_get_info()[0] == before


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
