"""Which small systems the shared-memory CG takes: a numbering whose column windows
span everything needs the window of p alone, as much as a replica of p."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sps

from jfem_b200 import _native as N


def windows(n, nnz, win):
    f = N.load()["_ZN3jfg16cg_small_windowsEiii"]
    f.restype, f.argtypes = C.c_int, [C.c_int] * 3
    return f(n, nnz, win)


@pytest.mark.parametrize("per_row", [3, 5, 9, 25])
def test_every_numbering_that_a_replica_of_p_fits(per_row):
    for n in range(1, 16400, 83):
        R = -(-n // 8)
        nnz = R * per_row
        replica = R <= 2048 and 8 * (n + nnz) + 4 * (R + 1 + nnz) + 16 <= 200 * 1024
        assert (windows(n, nnz, n) > 0) == replica, n          # no band at all
        assert windows(n, nnz, min(n, R + 200)) >= windows(n, nnz, n)
    assert windows(8000, 9000, 8000) == 1 and windows(4225, 4800, 800) == 2


def grid_laplace(m, rng):
    """9-point operator of an m x m grid, its unknowns in a random order."""
    one = sps.diags([np.ones(m - 1), np.ones(m), np.ones(m - 1)], [-1, 0, 1])
    A = (9.2 * sps.identity(m * m) - sps.kron(one, one)).tocsr()
    if rng is not None:
        q = rng.permutation(m * m)
        A = A[q][:, q]
    return A.tocoo()


@pytest.mark.gpu
@pytest.mark.parametrize("m", [80, 85, 90, 96])               # one window at 7,225 to 9,216 rows
def test_random_numbering(ctx, monkeypatch, m):
    from jfem_b200.linalg import DeviceMatrix, IterativeSolver

    rng = np.random.default_rng(m)
    A = grid_laplace(m, rng)
    b = rng.standard_normal(m * m)
    M = DeviceMatrix(m * m, m * m, A.row, A.col, A.data, ctx)
    its = []
    for small in ("1", "0"):
        monkeypatch.setenv("JFEM_SMALL_CG", small)
        s = IterativeSolver(ctx=ctx)
        x = s.solveCG(M, b, 1e-9)
        its.append(s.iterations)
        assert s.last.status == N.OK and np.linalg.norm(A @ x - b) < 1e-8
    assert abs(its[0] - its[1]) <= 1


@pytest.mark.gpu
@pytest.mark.parametrize("m", [3, 17, 65, 80])
def test_one_window_is_the_same_bits(ctx, monkeypatch, m):
    from jfem_b200.linalg import DeviceMatrix, IterativeSolver

    rng = np.random.default_rng(m)
    A = grid_laplace(m, None)
    b = rng.standard_normal(m * m)
    M = DeviceMatrix(m * m, m * m, A.row, A.col, A.data, ctx)
    out = []
    for mode in ("2", "p"):
        monkeypatch.setenv("JFEM_SMALL_CG_SMEM", mode)
        s = IterativeSolver(ctx=ctx)
        out.append((s.solveCG(M, b, 1e-11), s.iterations))
    assert out[0][1] == out[1][1] and np.array_equal(out[0][0], out[1][0])
