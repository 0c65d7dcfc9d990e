"""Kernel attributes belong to a device: what is set once is set once per device, not
once per process (a second device would launch without the opt-in shared memory)."""
import os
import re
import shutil
import subprocess

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "jfem_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

# jfg_per_device.h over a runtime of three devices that exists here only
HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <thread>
#include <vector>
#include "jfg_per_device.h"

static thread_local int current = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); std::exit(1); } } while (0)

int main()
{
    static jfg::PerDevice a, b;
    int calls[3] = {0, 0, 0};
    auto f = [&] { calls[current]++; return 10 + current; };
    for (int round = 0; round < 3; round++)
        for (int d : {1, 0, 2}) {
            current = d;
            CHECK(a.get(f) == 10 + d);
        }
    CHECK(calls[0] == 1 && calls[1] == 1 && calls[2] == 1);
    current = 1;                                    // a failure is not kept
    int tries = 0;
    auto g = [&]() -> int { if (tries++ == 0) throw std::runtime_error("no"); return 0; };
    bool thrown = false;
    try { b.get(g); } catch (const std::runtime_error&) { thrown = true; }
    CHECK(thrown && b.get(g) == 0 && b.get(g) == 0 && tries == 2);
    static jfg::PerDevice c;                        // many threads: one call per device
    std::atomic<int> n[2];
    n[0] = n[1] = 0;
    std::vector<std::thread> ts;
    for (int t = 0; t < 16; t++)
        ts.emplace_back([&, t] {
            current = t % 2;
            for (int k = 0; k < 1000; k++) CHECK(c.get([&] { n[current]++; return 7 + current; }) == 7 + t % 2);
        });
    for (auto& t : ts) t.join();
    CHECK(n[0] == 1 && n[1] == 1);
    return 0;
}
"""


def test_value_per_device(tmp_path):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")):
        pytest.skip("no host compiler or no CUDA headers")
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.check_call(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-I", os.path.join(CUDA, "include"), "-o", str(exe),
                           str(src)])
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).returncode == 0


def test_no_attribute_behind_a_static_of_the_process():
    bad = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, f)) as h:
            lines = h.read().split("\n")
        for i, line in enumerate(lines):
            if re.search(r"\b(cudaFuncSetAttribute|resident_cluster)\(", line):
                near = "\n".join(lines[max(0, i - 6):i + 1])
                if re.search(r"\bstatic\s+(const\s+)?(bool|int)\s+\w+\s*=", near):
                    bad.append((f, i + 1))
    assert not bad, bad


@pytest.mark.gpu
def test_second_device():
    """Blocked LU, its one-right-hand-side solve and a small CG on device 1 after device 0."""
    if torch.cuda.device_count() < 2:
        pytest.skip("one device")
    import numpy as np

    from jfem_b200 import _native as N
    from jfem_b200.linalg import DenseMatrix, DeviceMatrix, IterativeSolver

    rng = np.random.default_rng(5)
    A, b = rng.standard_normal((300, 300)) + 40 * np.eye(300), rng.standard_normal(300)
    i = np.arange(4000)
    for d in (0, 1, 0):
        ctx = N.Context(d)
        assert np.allclose(A @ DenseMatrix(A, ctx=ctx).solve(b), b, rtol=0, atol=1e-10)
        M = DeviceMatrix(4000, 4000, i, i, 1.0 + i % 3, ctx)
        s = IterativeSolver(ctx=ctx)
        assert np.allclose(s.solveCG(M, np.ones(4000), 1e-12), 1.0 / (1.0 + i % 3), rtol=0, atol=1e-10)
