"""Device blocks kept between owners: bounded, given back, and safe for
contexts in several threads."""
import threading

import numpy as np
import pytest
import torch

from jfem_b200 import _native as N
from jfem_b200.linalg import DeviceMatrix

pytestmark = pytest.mark.gpu


def triples(n, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    r = np.concatenate([i, i[1:], i[:-1]])
    c = np.concatenate([i, i[:-1], i[1:]])
    return r, c, rng.standard_normal(r.size)


def test_pool_is_bounded_and_given_back():
    ctx = N.Context(0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for k in range(12):                                  # ~150 MB each, of ever larger classes
        n = 1_000_000 + 120_000 * k
        DeviceMatrix(n, n, *triples(n, k), ctx)          # dropped at once
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= (1 << 30) + (64 << 20), kept          # the bound, and the driver's own granularity
    ctx.check(N.load().jfg_release_scratch(ctx.handle))
    assert before - torch.cuda.mem_get_info()[0] <= 64 << 20


def test_threads_with_their_own_contexts():
    def work(seed, out):
        ctx = N.Context(0)
        for k in range(8):
            n = 3000 + 517 * k
            r, c, v = triples(n, seed + k)
            A = DeviceMatrix(n, n, r, c, v, ctx)
            x = np.random.default_rng(seed - k).standard_normal(n)
            y = np.zeros(n)
            np.add.at(y, r, v * x[c])
            # three products per row: at most a few roundings of their absolute sum
            s = np.zeros(n)
            np.add.at(s, r, np.abs(v * x[c]))
            out.append(bool(np.all(np.abs(A.spmv(x) - y) <= 4 * 2.0 ** -52 * s)))
            del A
        ctx.close()

    outs = [[] for _ in range(4)]
    ts = [threading.Thread(target=work, args=(100 * (i + 1), outs[i])) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert all(len(o) == 8 and all(o) for o in outs)
