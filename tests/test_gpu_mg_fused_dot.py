"""The FP64 PCG whose r . z is summed by the multigrid's last sweep."""
import numpy as np
import pytest

from fixtures import coo_oracle, mg_levels
from jfem_b200 import IterativeSolver, JacobiSmoother, MGPreconditioner
from jfem_b200.linalg import DeviceMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,coarse,L,runs,cycles,boundary", [
    (1, 3, 2, 2, 1, "once"),      # 49 rows: less than one block of the sweep
    (1, 5, 4, 1, 1, "once"),
    (1, 5, 4, 3, 2, "once"),      # only the last of two cycles forms the dot
    (2, 3, 4, 2, 1, "once"),      # SELL-32 rows
    (1, 5, 4, 2, 1, "none"),      # no boundary list on the finest level: the dot stays a pass of its own
    (1, 5, 4, 2, 1, "twice"),     # an unknown named twice counts once
])
def test_pcg_matches_numpy(ctx, p, coarse, L, runs, cycles, boundary):
    """Residual history and solution against the PCG in NumPy with
    the device's preconditioner: the dots differ
    by their summation order only (n * 1.1e-16 < 1e-12 of the sum of
    magnitudes), which the at most 30 iterations of a preconditioner with
    contraction below 0.3 carry on without growth beyond the factor 1e3
    between an iteration's change and its residual: 1e-9 of the first norm."""
    h = mg_levels(p, coarse, L, modes=8, seed=2)
    b = h.finest.rhs
    bd = [np.asarray(q) for q in h.boundary]
    if boundary == "none":
        bd[-1] = np.zeros(0, bd[-1].dtype)
    elif boundary == "twice":
        bd[-1] = np.concatenate([bd[-1], bd[-1][:1]])
    mats = [DeviceMatrix(s.n, s.n, s.rows, s.cols, s.vals, ctx) for s in h.systems]
    prol = [DeviceMatrix(h.systems[l + 1].n, h.systems[l].n, *h.prolong[l], ctx) for l in range(L - 1)]
    mg = MGPreconditioner(mats, prol, bd, [None] + [JacobiSmoother(runs, 2.0 / 3.0)] * (L - 1), cycles=cycles,
                          use_fmg=False, ctx=ctx)
    s = IterativeSolver(ctx=ctx)
    s.precision = "fp64"
    x = s.solvePCG(mats[-1], mg, b, 1e-9 * np.linalg.norm(b))
    A = coo_oracle(h.finest)
    dense = A.dense()
    assert np.linalg.norm(b - dense @ x) <= 2e-9 * np.linalg.norm(b)
    # the same iteration in NumPy with the device's preconditioner, from the first unit vector
    xo = np.zeros_like(b)
    xo[0] = 1.0
    r = b - dense @ xo
    z = mg.mvMul(r)
    pv = z.copy()
    rz = r @ z
    hist = [np.linalg.norm(r)]
    for _ in range(s.iterations):
        Ap = dense @ pv
        al = rz / (pv @ Ap)
        xo = xo + al * pv
        r = r - al * Ap
        hist.append(np.linalg.norm(r))
        z = mg.mvMul(r)
        rz, old = r @ z, rz
        pv = z + (rz / old) * pv
    got = np.asarray(s.last.history)[: s.iterations]
    want = np.asarray(hist[1: 1 + got.size])
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-9 * hist[0])
    np.testing.assert_allclose(x, xo, rtol=0, atol=1e-9 * np.abs(xo).max())
