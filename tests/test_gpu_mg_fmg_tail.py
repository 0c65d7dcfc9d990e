"""Full multigrid on the coarse levels in one cluster launch (k_mg_tail<T, true>)."""
import numpy as np
import pytest

import oracle as O
from fixtures import coo_oracle, mg_levels
from jfem_b200 import JacobiSmoother, MGPreconditioner
from jfem_b200.linalg import DeviceMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,coarse,L,runs", [
    (1, 4, 2, 2),     # no level between the coarsest and the finest: no tail
    (1, 4, 3, 2),     # every tail level owned by one CTA
    (1, 4, 6, 1),     # one sweep: the sweep from the prolongation ends in the spare vector and is copied
    (1, 3, 6, 2),
    (1, 5, 6, 3),
    (2, 2, 6, 2),
    (1, 7, 7, 2),     # tail levels spread over the cluster, several levels above it
])
def test_fmg_tail_matches_per_launch(ctx, monkeypatch, p, coarse, L, runs):
    """Same operations per row in both paths; only the order of the up to 25
    products of a row sum differs (column order, or 4 partial sums), so each
    of the at most 400 dependent row operations of a scheme on up to 7 levels
    differs by at most 25 * 1.1e-16 of the row's terms: 1.1e-12 of the largest
    value with no growth, 1e-10 with the factor 100 that the residuals'
    cancellation may add."""
    h = mg_levels(p, coarse, L, modes=8, seed=11)
    b = h.finest.rhs
    outs = []
    for tail, local in (("1", "1"), ("1", "0"), ("0", "1")):
        monkeypatch.setenv("JFEM_MG_TAIL", tail)
        monkeypatch.setenv("JFEM_MG_TAIL_LOCAL", local)
        mats = [DeviceMatrix(s.n, s.n, s.rows, s.cols, s.vals, ctx) for s in h.systems]
        prol = [DeviceMatrix(h.systems[l + 1].n, h.systems[l].n, *h.prolong[l], ctx) for l in range(L - 1)]
        mg = MGPreconditioner(mats, prol, h.boundary, [None] + [JacobiSmoother(runs, 2.0 / 3.0)] * (L - 1), cycles=1,
                              use_fmg=True, ctx=ctx)
        outs.append(mg.mvMul(b))
    assert np.all(np.isfinite(outs[0]))
    assert np.array_equal(outs[0], outs[1])
    np.testing.assert_allclose(outs[0], outs[2], rtol=0, atol=1e-10 * np.abs(outs[2]).max())
    if L < 7:
        prol_o = [O.CooMatrix(h.systems[l + 1].n, h.systems[l].n, *h.prolong[l]) for l in range(L - 1)]
        mg_o = O.MGPreconditioner([coo_oracle(s) for s in h.systems], prol_o, h.boundary,
                                  [None] + [(O.SMOOTH_JACOBI, runs, 2.0 / 3.0)] * (L - 1), cycles=1, use_fmg=True)
        ref = mg_o.mvmul(b)
        np.testing.assert_allclose(outs[0], ref, rtol=0, atol=1e-10 * np.abs(ref).max())
