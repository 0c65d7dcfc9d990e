"""Coloured Schwarz sweeps of a level in one cooperative launch against one
launch per colour: the same sums in the same order, so the same bits -- one
patch per CTA, several patches per batch, fewer patches than colours, one and
more runs, FP64 and FP32 hierarchies, inverses in shared and global memory."""
import numpy as np
import pytest

from jfem_b200.linalg import DeviceMatrix
from jfem_b200.schwarz import ColoredCartesianSchwarz, DirectSolver, SchwarzSmoother
from jfem_b200.stokes import MonolithicStokesMG, StokesSolver, TaylorHoodSpace, stokes_problem, velocity_block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,partitions,overlap", [(4, 2, 1), (8, 4, 1), (24, 12, 1), (32, 16, 1), (72, 36, 1)])
@pytest.mark.parametrize("runs", [1, 3])
def test_sweep_equals_colour_launches(ctx, monkeypatch, cells, partitions, overlap, runs):
    th = TaylorHoodSpace(cells, cells)
    R, Cc, V, _ = velocity_block(th)
    A = DeviceMatrix(th.nv, th.nv, R, Cc, V, ctx)
    rng = np.random.default_rng(51)
    b, x = rng.standard_normal(th.nv), rng.standard_normal(th.nv)
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("JFEM_SCHWARZ_SWEEP", flag)
        sw = ColoredCartesianSchwarz(A, th.velocity, (partitions, partitions), overlap, DirectSolver(), 0.9)
        sm = SchwarzSmoother(runs, sw)
        out.append([sm.smooth(A, b, x), sm.smooth(A, x, b)])      # the handle is reused
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("fp32", [False, True])
def test_sweep_in_the_velocity_v_cycle(ctx, monkeypatch, fp32):
    prob = stokes_problem(24, 3, seed=2, pin_pressure=False)
    v = np.random.default_rng(52).standard_normal(prob.system.n)
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("JFEM_SCHWARZ_SWEEP", flag)
        S = StokesSolver(ctx, prob, fp32_vcycle=fp32)
        out.append((S.P.mvMul(v), S.solve(1e-8)[0]))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_sweep_with_inverses_in_global_memory(ctx, monkeypatch):
    v = out = None
    res = []
    for flag in ("1", "0"):
        monkeypatch.setenv("JFEM_SCHWARZ_SWEEP", flag)
        S = MonolithicStokesMG(ctx, cells=16, coarse_cells=4, seed=3)
        v = np.random.default_rng(53).standard_normal(S.A.rows)
        res.append(S.mg.mvMul(v))
    assert np.array_equal(res[0], res[1])
