"""Small batches of small systems: wide clusters in the on-chip heat kernel.

Rows are dealt to CTAs in whole warps, so a wide cluster of a small system may
have more CTAs than rows to deal, and the threads past a CTA's last row read the
halo words beside it.  No CTA may be without rows, and what a kernel before left
in shared memory may not reach the result."""
import numpy as np
import pytest

from jfem_b200.assembly import Space, assemble_device
from jfem_b200.batch import BatchedParabolicIntegrator

pytestmark = pytest.mark.gpu


def systems(ctx, cells, count):
    sp = Space(1, cells, cells)
    K = [assemble_device(sp, 1e-3 * (1 + s), 1.0, dirichlet=False, ctx=ctx)[0] for s in range(count)]
    M = [assemble_device(sp, 0.0, 1.0, dirichlet=False, ctx=ctx)[0]] * count
    px, py = sp.node_points()
    u = [np.cos(3 * px + s) * np.sin(2 * py) for s in range(count)]
    return sp, K, M, u


def leave_nans(ctx):
    """A batch of NaN states over every SM: it stops at its first residual, whose
    NaN stay in shared memory."""
    sp, K, M, _ = systems(ctx, 16, 1)
    count = 148 * 8
    B = BatchedParabolicIntegrator(K * count, M * count, ctx)
    B.timeSteps([np.full(sp.n, np.nan)] * count, 1)
    assert B.last.failed == count


@pytest.mark.parametrize("cells", [16, 20, 24, 32, 40, 64])
@pytest.mark.parametrize("count", [1, 4, 9, 18])
def test_every_cta_owns_a_row(ctx, cells, count):
    sp, K, M, u = systems(ctx, cells, count)
    B = BatchedParabolicIntegrator(K, M, ctx)
    B.timeSteps(u, 1)
    C = B.last.cluster
    rows = -(-(-(-sp.n // C)) // 32) * 32            # of a CTA: the even share in whole warps
    assert B.last.failed == 0 and (C - 1) * rows < sp.n, (C, rows, sp.n)


@pytest.mark.parametrize("cells", [16, 20, 24, 32, 40, 64])
@pytest.mark.parametrize("count", [1, 4])
def test_what_was_in_shared_memory_does_not_matter(ctx, cells, count):
    sp, K, M, u = systems(ctx, cells, count)
    B = BatchedParabolicIntegrator(K, M, ctx)
    leave_nans(ctx)
    a = B.timeSteps(u, 2)
    assert B.last.status == 0 and B.last.failed == 0
    leave_nans(ctx)
    assert np.array_equal(B.timeSteps(u, 2), a)
    b = B.timeSteps(u, 2, cluster=2, threads=256, rows_per_thread=2)
    # both solve every step to a 1e-10 relative residual
    for x, y in zip(B.unpack(a), B.unpack(b)):
        assert np.linalg.norm(x - y) < 1e-8 * np.linalg.norm(y)
