"""A coloured Schwarz sweep whose CTAs do not meet: the wait is bounded, the call
says so, and the handle is good again afterwards.  Zero polls make every wait run
out at once, on every path that smooths with the sweep."""
import numpy as np
import pytest

from jfem_b200 import _native as N
from jfem_b200.linalg import DeviceMatrix
from jfem_b200.schwarz import ColoredCartesianSchwarz, DirectSolver, SchwarzSmoother
from jfem_b200.stokes import MonolithicStokesMG, StokesSolver, TaylorHoodSpace, stokes_problem, velocity_block

pytestmark = pytest.mark.gpu


def runs_out(monkeypatch, call):
    monkeypatch.setenv("JFEM_SCHWARZ_SWEEP_SPINS", "0")
    with pytest.raises(N.JfgError, match="ran out") as e:
        call()
    assert e.value.status == N.ERR_CUDA
    monkeypatch.delenv("JFEM_SCHWARZ_SWEEP_SPINS")


@pytest.mark.parametrize("cells,partitions", [(4, 2), (24, 12), (32, 16)])
def test_smoothing(ctx, monkeypatch, cells, partitions):
    th = TaylorHoodSpace(cells, cells)
    R, Cc, V, _ = velocity_block(th)
    A = DeviceMatrix(th.nv, th.nv, R, Cc, V, ctx)
    rng = np.random.default_rng(61)
    b, x = rng.standard_normal(th.nv), rng.standard_normal(th.nv)
    sw = ColoredCartesianSchwarz(A, th.velocity, (partitions, partitions), 1, DirectSolver(), 0.9)
    sm = SchwarzSmoother(2, sw)
    good = sm.smooth(A, b, x)
    for _ in range(2):
        runs_out(monkeypatch, lambda: sm.smooth(A, b, x))
        assert np.array_equal(sm.smooth(A, b, x), good)
    monkeypatch.setenv("JFEM_SCHWARZ_SWEEP", "0")
    plain = ColoredCartesianSchwarz(A, th.velocity, (partitions, partitions), 1, DirectSolver(), 0.9)
    assert np.array_equal(SchwarzSmoother(2, plain).smooth(A, b, x), good)


def test_v_cycle_and_solve(ctx, monkeypatch):
    prob = stokes_problem(24, 3, seed=2, pin_pressure=False)
    v = np.random.default_rng(62).standard_normal(prob.system.n)
    S = StokesSolver(ctx, prob)
    z = S.P.mvMul(v)
    runs_out(monkeypatch, lambda: S.P.mvMul(v))
    assert np.array_equal(S.P.mvMul(v), z)
    runs_out(monkeypatch, lambda: StokesSolver(ctx, prob).solve(1e-8))
    x = S.solve(1e-8)[0]
    assert np.all(np.isfinite(x)) and np.array_equal(S.P.mvMul(v), z)


def test_inverses_in_global_memory(ctx, monkeypatch):
    S = MonolithicStokesMG(ctx, cells=16, coarse_cells=4, seed=3)
    v = np.random.default_rng(63).standard_normal(S.A.rows)
    z = S.mg.mvMul(v)
    runs_out(monkeypatch, lambda: S.mg.mvMul(v))
    assert np.array_equal(S.mg.mvMul(v), z)


@pytest.mark.parametrize("cells,partitions", [(24, 12), (72, 36)])   # CTAs without a batch in some colours
def test_waits_that_run_out_at_different_steps(ctx, monkeypatch, cells, partitions):
    """Few polls: CTAs give up at different steps, each as a whole.  Every call ends,
    with the usual bits or with the error."""
    th = TaylorHoodSpace(cells, cells)
    R, Cc, V, _ = velocity_block(th)
    A = DeviceMatrix(th.nv, th.nv, R, Cc, V, ctx)
    rng = np.random.default_rng(64)
    b, x = rng.standard_normal(th.nv), rng.standard_normal(th.nv)
    sm = SchwarzSmoother(3, ColoredCartesianSchwarz(A, th.velocity, (partitions, partitions), 1, DirectSolver(), 0.9))
    good = sm.smooth(A, b, x)
    ends = {"bits": 0, "error": 0}
    for spins in (1, 2, 3, 5, 8, 12, 20, 40) * 4:
        monkeypatch.setenv("JFEM_SCHWARZ_SWEEP_SPINS", str(spins))
        try:
            assert np.array_equal(sm.smooth(A, b, x), good)
            ends["bits"] += 1
        except N.JfgError as e:
            assert e.status == N.ERR_CUDA and "ran out" in str(e)
            ends["error"] += 1
    monkeypatch.delenv("JFEM_SCHWARZ_SWEEP_SPINS")
    assert ends["error"] > 0 and np.array_equal(sm.smooth(A, b, x), good)
