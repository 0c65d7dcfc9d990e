"""Releases while a stream of the device is being captured, as plain cudaFree
allows them: neither the capture nor the releasing thread may notice."""
import threading

import numpy as np
import pytest
import torch

from jfem_b200 import _native as N
from jfem_b200.linalg import DeviceMatrix, IterativeSolver

pytestmark = pytest.mark.gpu


def laplace(ctx, n, shift):
    i = np.arange(n)
    r = np.concatenate([i, i[1:], i[:-1]])
    c = np.concatenate([i, i[:-1], i[1:]])
    v = np.concatenate([np.full(n, 2.0 + shift), np.full(2 * n - 2, -1.0)])
    return DeviceMatrix(n, n, r, c, v, ctx), (r, c, v)


def build_and_drop(ctx, n):
    A, (r, c, v) = laplace(ctx, n, 0.5)
    x = np.cos(np.arange(n))
    y = np.zeros(n)
    np.add.at(y, r, v * x[c])
    assert np.allclose(A.spmv(x), y, rtol=0, atol=1e-13)
    del A


@pytest.mark.parametrize("library_stream", [False, True])
def test_release_during_a_capture_of_another_thread(library_stream):
    own, other = N.Context(0), N.Context(0)
    dev = torch.device("cuda", 0)
    st = torch.cuda.ExternalStream(N.load().jfg_stream(other.handle)) if library_stream else torch.cuda.Stream(dev)
    x = torch.zeros(1000, device=dev)
    torch.cuda.synchronize()
    capturing, dropped, errors = threading.Event(), threading.Event(), []

    def capture():
        try:
            with torch.cuda.stream(st):
                g = torch.cuda.CUDAGraph()
                g.capture_begin(capture_error_mode="thread_local")
                x.add_(1.0)
                capturing.set()
                dropped.wait(60)
                x.add_(2.0)
                g.capture_end()
                g.replay()
                st.synchronize()
        except Exception as e:                       # noqa: BLE001 -- handed to the test
            errors.append(e)
        finally:
            capturing.set()

    build_and_drop(own, 4000)                        # the library's kernels are loaded before the capture
    t = threading.Thread(target=capture)
    t.start()
    capturing.wait(60)
    try:
        for k in range(3):
            build_and_drop(own, 5000 + 700 * k)
    finally:
        dropped.set()
        t.join()
    assert not errors and float(x.sum()) == 3000.0
    build_and_drop(own, 9000)


def test_solves_that_capture_beside_releases():
    errors, stop = [], threading.Event()

    def solve(seed):
        try:
            ctx = N.Context(0)
            for k in range(30):                      # a new matrix each: its iteration is captured anew
                n = 20000 + 64 * k
                A, _ = laplace(ctx, n, 0.5)
                b = np.random.default_rng(seed + k).standard_normal(n)
                s = IterativeSolver(ctx=ctx)
                x = s.solveCG(A, b, 1e-8)
                assert s.last.status == N.OK and np.linalg.norm(A.spmv(x) - b) < 1e-7
                del A
            ctx.close()
        except Exception as e:                       # noqa: BLE001
            errors.append(e)

    def drop():
        try:
            ctx = N.Context(0)
            k = 0
            while not stop.is_set():
                build_and_drop(ctx, 3000 + 100 * (k % 7))
                k += 1
            ctx.close()
        except Exception as e:                       # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=solve, args=(10 * i,)) for i in range(2)]
    ds = [threading.Thread(target=drop) for _ in range(2)]
    for t in ts + ds:
        t.start()
    for t in ts:
        t.join()
    stop.set()
    for t in ds:
        t.join()
    assert not errors, errors
