"""The first solve of a context: its device blocks may hold what their last owner
left, and the legacy stream may be busy with other work of the process."""
import numpy as np
import pytest
import torch

from jfem_b200 import _native as N
from jfem_b200.linalg import DeviceMatrix, IterativeSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [500, 40000])
def test_first_solve_on_used_blocks(n):
    first = N.Context(0)
    keep = [DeviceMatrix(5, 5, np.arange(5), np.arange(5), np.full(5, -7.5 - k), first) for k in range(24)]
    del keep                                         # small blocks, none of them zero
    i = np.arange(n)
    r = np.concatenate([i, i[1:], i[:-1]])
    c = np.concatenate([i, i[:-1], i[1:]])
    v = np.concatenate([np.full(n, 2.5), np.full(2 * n - 2, -1.0)])
    b = np.sin(i + 1.0)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)                   # ~0.1 s on the legacy stream
    ctx = N.Context(0)
    A = DeviceMatrix(n, n, r, c, v, ctx)
    s = IterativeSolver(ctx=ctx)
    x = s.solveCG(A, b, 1e-9)
    y = np.zeros(n)
    np.add.at(y, r, v * x[c])
    assert s.last.status == N.OK and np.linalg.norm(y - b) < 1e-8
