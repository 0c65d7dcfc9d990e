"""Batched heat systems in the on-chip kernel (K in shared memory, vectors in
registers, one cluster per system) against the general kernel, at the edges of
its variants (rows per CTA), cluster sizes, odd and even grid strides, together
with systems only the general kernel takes."""
import numpy as np
import pytest

from jfem_b200.assembly import Space, assemble_device
from jfem_b200.batch import BatchedParabolicIntegrator

pytestmark = pytest.mark.gpu

# 441 ... 1,536 | 1,560 ... 4,556 rows in one CTA, then two and more; (9, 9) has no 9-point layout
GRIDS = [(20, 20), (15, 31), (38, 38), (39, 38), (67, 66), (68, 66), (131, 70), (9, 9), (150, 143)]


@pytest.mark.parametrize("copies", [1, 8])
@pytest.mark.parametrize("source", [False, True])
def test_onchip_matches_general_kernel(ctx, copies, source):
    rng = np.random.default_rng(41)
    K, M, u, f = [], [], [], []
    for cx, cy in GRIDS * copies:
        sp = Space(1, cx, cy)
        dt = 1e-3 * (1 + rng.random())
        kappa = np.exp(rng.standard_normal(cx * cy))
        K.append(assemble_device(sp, dt, 1.0, grad_coef_cells=kappa, dirichlet=False, ctx=ctx)[0])
        M.append(assemble_device(sp, 0.0, 1.0, dirichlet=False, ctx=ctx)[0])
        px, py = sp.node_points()
        u.append(np.cos(3 * px) * np.sin(2 * py + rng.random()) + rng.standard_normal(sp.n) * 0.1)
        f.append(1e-3 / sp.n * rng.standard_normal(sp.n))
    B = BatchedParabolicIntegrator(K, M, ctx)
    fs = f if source else None
    a = B.timeSteps(u, 3, fs)
    assert B.last.status == 0 and B.last.failed == 0 and B.last.max_rel_residual <= 1e-10
    b = B.timeSteps(u, 3, fs, cluster=4, threads=512, rows_per_thread=3)
    assert B.last.failed == 0
    # both solve every step to a 1e-10 relative residual
    for x, y in zip(B.unpack(a), B.unpack(b)):
        assert np.linalg.norm(x - y) < 1e-8 * np.linalg.norm(y)


def test_onchip_reports_failures(ctx):
    sp = Space(1, 40, 40)
    K = [assemble_device(sp, 1e-3, 1.0, dirichlet=False, ctx=ctx)[0] for _ in range(3)]
    M = [assemble_device(sp, 0.0, 1.0, dirichlet=False, ctx=ctx)[0] for _ in range(3)]
    B = BatchedParabolicIntegrator(K, M, ctx)
    u = [np.ones(sp.n), np.full(sp.n, np.nan), np.ones(sp.n)]
    B.timeSteps(u, 2)
    assert B.last.status == 3 and B.last.failed == 1
    v = [np.cos(7 * sp.node_points()[0]), np.zeros(sp.n), np.ones(sp.n)]
    w = B.unpack(B.timeSteps(v, 2, max_refine=0, rtol=1e-14))
    # only the first needs a refinement: zero is solved, and a constant is steady (K 1 = M 1)
    assert B.last.failed == 1 and np.array_equal(w[1], v[1])
