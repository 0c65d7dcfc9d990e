"""Performance cases: the work a user of jfem_b200 has the library do.

Every case goes through the public entry points (``jfem_b200.linalg``,
``multigrid``, ``cnn``, ``batch``, ``stokes``).  ``listed()`` names the fixed
cases, ``draw(rng)`` makes further ones of the same ranges, ``prepare`` makes
what a user's program holds before the call, ``run`` is one call, ``work`` the
bytes and operations the call cannot do without, and ``exact`` the same result
in plain 64-bit torch.

Kinds:
  cg        unpreconditioned FP64 CG of a Q1 system (the small drop-in solve)
  pcg       CG preconditioned by the geometric multigrid V-cycle (Jacobi 2 + 2):
            FP64, FP32 V-cycle, or a V-cycle reading scaled-FP16 matrices
  fgmres    FGMRES(30) with the FP32 V-cycle and the learned smoother
  mgapply   the reference's preconditioner (FMG + 3 V-cycles) on host vectors
  cnngrad   loss and weight gradient of the learned smoother (one training step's device work)
  heat      batched implicit Euler of many uneven systems
  stokes    Taylor-Hood Stokes, GMRES(50), Schwarz- or Jacobi-smoothed velocity multigrid
  dense     dense LU solve of host data
  galerkin  coarse operator P^T A P, read back as CSR
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

from jfem_b200 import _native as N
from jfem_b200.assembly import Space, assemble_device, prolongation
from jfem_b200.batch import BatchedParabolicIntegrator
from jfem_b200.cnn import SHAPES, LearnedSmoother, MGCNNPreconditioner, he_init, pixel_map
from jfem_b200.learned import WEIGHTS
from jfem_b200.linalg import DenseMatrix, DeviceMatrix, IterativeSolver
from jfem_b200.multigrid import JacobiSmoother, MGPreconditioner
from jfem_b200.stokes import StokesSolver, stokes_problem

CORR_LENGTH = 0.05          # of the log-normal coefficient
GRID_PRECISION = {"fp64": "fp64", "mixed": "mixed-precond", "mixed-fp16": "mixed-precond"}


def listed():
    return [
        # the smallest solve: one call of solveCG, bound by latency
        {"name": "cg_q1_64", "kind": "cg", "cells": 64},
        # the reference's own preconditioner call on host vectors, an odd coarse grid (225 x 225 nodes)
        {"name": "mgapply_q1_224", "kind": "mgapply", "p": 1, "coarse": 7, "levels": 6},
        # an ordinary solve, 193 x 193 nodes, every digit in FP64
        {"name": "pcg_q1_192_fp64", "kind": "pcg", "p": 1, "coarse": 3, "levels": 7, "kappa": False,
         "precision": "fp64"},
        # the benchmark system (kappa = exp of a Gaussian field, 1025 x 1025 nodes): the drop-in solve ...
        {"name": "pcg_q1_1024_fp64", "kind": "pcg", "p": 1, "coarse": 4, "levels": 9, "kappa": True,
         "precision": "fp64"},
        # ... and with the FP32 V-cycle
        {"name": "pcg_q1_1024_mixed", "kind": "pcg", "p": 1, "coarse": 4, "levels": 9, "kappa": True,
         "precision": "mixed"},
        # Q2 elements (general sparse rows), V-cycle matrices stored in FP16
        {"name": "pcg_q2_512_fp16", "kind": "pcg", "p": 2, "coarse": 4, "levels": 8, "kappa": False,
         "precision": "mixed-fp16"},
        # the headline solve: FGMRES(30), FP32 V-cycle and the learned smoother
        {"name": "fgmres_learned_1024", "kind": "fgmres", "coarse": 4, "levels": 9},
        # the training step's gradient on a batch of crops
        {"name": "cnngrad_16x128x128", "kind": "cnngrad", "batch": 16, "height": 128, "width": 128},
        # many uneven heat systems, ten implicit-Euler steps
        {"name": "heat_96x10", "kind": "heat", "systems": 96, "min_cells": 32, "max_cells": 256, "steps": 10},
        # lid-driven cavity, Taylor-Hood, coloured Schwarz smoothing
        {"name": "stokes_64_schwarz", "kind": "stokes", "coarse": 4, "levels": 5, "smoother": "schwarz"},
        # dense direct solve of host data, a ragged size
        {"name": "dense_2049", "kind": "dense", "n": 2049},
        # Galerkin coarse operator of a Q1 coefficient problem, 513 x 513 nodes
        {"name": "galerkin_q1_512", "kind": "galerkin", "cells": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo_cells, hi_cells):
    """(coarse, levels) with lo_cells <= coarse * 2^(levels - 1) <= hi_cells."""
    while True:
        coarse = rng.randint(3, 7)
        levels = rng.randint(3, 9)
        if lo_cells <= coarse << (levels - 1) <= hi_cells:
            return coarse, levels


def draw(rng):
    kind = rng.choice(["cg", "mgapply", "pcg", "pcg", "pcg", "fgmres", "cnngrad", "heat", "stokes", "dense",
                       "galerkin"])
    case = {"kind": kind}
    if kind == "cg":
        case.update(cells=_log_int(rng, 16, 300))
    elif kind == "mgapply":
        coarse, levels = _grid(rng, 24, 448)
        case.update(p=1, coarse=coarse, levels=levels)
    elif kind == "pcg":
        p = rng.choice([1, 1, 2])
        coarse, levels = _grid(rng, 48, 1024 // p)
        case.update(p=p, coarse=coarse, levels=levels, kappa=rng.random() < 0.5,
                    precision=rng.choice(["fp64", "mixed", "mixed-fp16"]))
    elif kind == "fgmres":
        coarse, levels = _grid(rng, 96, 1024)
        case.update(coarse=coarse, levels=levels)
    elif kind == "cnngrad":
        height, width = _log_int(rng, 24, 512), _log_int(rng, 24, 512)
        case.update(batch=max(1, min(16, _log_int(rng, 1, 16), 600000 // (height * width))), height=height,
                    width=width)
    elif kind == "heat":
        lo = _log_int(rng, 16, 64)
        case.update(systems=_log_int(rng, 4, 96), min_cells=lo, max_cells=_log_int(rng, lo, 256),
                    steps=rng.randint(2, 10))
    elif kind == "stokes":
        coarse, levels = rng.choice([(3, 3), (4, 3), (5, 3), (3, 4), (4, 4), (5, 4), (6, 4), (7, 4), (4, 5)])
        case.update(coarse=coarse, levels=levels, smoother=rng.choice(["schwarz", "jacobi"]))
    elif kind == "dense":
        case.update(n=_log_int(rng, 40, 2100))
    else:
        case.update(cells=2 * _log_int(rng, 16, 256))
    return case


# ---------------------------------------------------------------------------
# inputs (from the seed alone)
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator()
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _kappa_cells(cells, seed):
    """exp of a Gaussian field with squared-exponential covariance at the cells (periodic sampling)."""
    n = 2 * cells
    idx = torch.arange(n, dtype=torch.float64, device="cuda")
    d = torch.minimum(idx, n - idx) / cells
    cov = torch.exp(-(d[:, None] ** 2 + d[None, :] ** 2) / (2 * CORR_LENGTH ** 2))
    lam = torch.fft.fft2(cov).real.clamp_min(0)
    w = torch.randn(n, n, generator=_generator(seed), dtype=torch.float64).cuda()
    g = torch.fft.ifft2(lam.sqrt() * torch.fft.fft2(w)).real[:cells, :cells]
    return torch.exp(g).cpu().numpy()


def _coarsen(k):
    return 0.25 * (k[0::2, 0::2] + k[1::2, 0::2] + k[0::2, 1::2] + k[1::2, 1::2])


def _load_grid(nodes, seed, modes):
    """Nodal load h^2 f on a nodes x nodes grid, f a sum of seeded sine modes; zero on the boundary."""
    a = torch.randn(modes, modes, generator=_generator(seed + 7919), dtype=torch.float64)
    t = torch.linspace(0, 1, nodes, dtype=torch.float64)
    s = torch.sin(math.pi * t[:, None] * torch.arange(1, modes + 1, dtype=torch.float64))
    f = (s @ a @ s.T) / (nodes - 1) ** 2
    f[0], f[-1], f[:, 0], f[:, -1] = 0, 0, 0, 0
    return f.numpy()


@lru_cache(maxsize=None)
def _space(p, cells):
    return Space(p, cells, cells)


@lru_cache(maxsize=None)
def _prolongation(p, cells):
    return prolongation(_space(p, cells), _space(p, 2 * cells))


def _problem(case, seed):
    """Coefficient per level (or None), mass coefficient and the load on the node grid."""
    p = case.get("p", 1)
    cells = case["coarse"] << (case["levels"] - 1)
    kappa = None
    if case.get("kappa", case["kind"] == "fgmres"):
        kappa = [_kappa_cells(cells, seed)]
        for _ in range(case["levels"] - 1):
            kappa.insert(0, _coarsen(kappa[0]))
    return p, cells, kappa, (0.0 if kappa else 5.0), _load_grid(p * cells + 1, seed, 16 if p == 2 else 4)


def _hierarchy(case, seed):
    p, cells, kappa, mass, load = _problem(case, seed)
    levels = case["levels"]
    mats, bds = [], []
    for l in range(levels):
        sp = _space(p, case["coarse"] << l)
        A, _, bd, _ = assemble_device(sp, 1.0, mass, grad_coef_cells=None if kappa is None else kappa[l])
        mats.append(A)
        bds.append(bd)
    prol = []
    for l in range(levels - 1):
        prol.append(DeviceMatrix(mats[l + 1].rows, mats[l].rows, *_prolongation(p, case["coarse"] << l)))
    rhs = np.empty(mats[-1].rows)
    rhs[_space(p, cells).node_of_grid] = load.reshape(-1)
    return mats, prol, bds, rhs


def _dense_inputs(n, seed):
    g = _generator(seed)
    a = torch.randn(n, n, generator=g, dtype=torch.float64)
    a.diagonal().add_(4 * math.sqrt(n))
    return a.numpy(), torch.randn(n, generator=g, dtype=torch.float64).numpy()


def _heat_inputs(case, seed):
    """Cells, time step and initial grid values (Gaussian bumps) of every system."""
    g = _generator(seed)
    sizes = torch.arange(case["min_cells"], case["max_cells"] + 1, 16)
    pick = sizes[torch.randint(0, len(sizes), (case["systems"],), generator=_generator(case["systems"]))]
    dt = 1e-3 * (1 + 0.1 * torch.rand(case["systems"], generator=g, dtype=torch.float64))
    u0 = []
    for c in pick.tolist():
        t = torch.linspace(0, 1, c + 1, dtype=torch.float64)
        r = torch.rand(4, 8, generator=g, dtype=torch.float64)
        cx, cy, s = 0.15 + 0.7 * r[0], 0.15 + 0.7 * r[1], 0.02 + 0.08 * r[2]
        ex = torch.exp(-(t[:, None] - cx) ** 2 / (2 * s * s))
        ey = torch.exp(-(t[:, None] - cy) ** 2 / (2 * s * s))
        u0.append((ex * (2 * r[3] - 1)) @ ey.T)
    return pick.tolist(), dt.tolist(), u0


def _images(case, seed):
    """Normalised residual images (white noise at unit rms) and smooth-scaled targets."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    shape = (case["batch"], case["height"], case["width"])
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
    t = 0.5 * torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
    return x, t, he_init(int(seed) & 0xFFFF, gain_last=0.5)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "cg":
        sp = _space(1, case["cells"])
        A, _, _, _ = assemble_device(sp, 1.0, 5.0)
        rhs = np.empty(sp.n)
        rhs[sp.node_of_grid] = _load_grid(sp.nx, seed, 4).reshape(-1)
        e0 = torch.zeros(sp.n, dtype=torch.float64, device="cuda")
        e0[0] = 1.0
        return {"kind": kind, "A": A, "b": torch.tensor(rhs, device="cuda"), "start": e0, "solver": IterativeSolver(),
                "tol": 1e-10 * float(np.linalg.norm(rhs))}
    if kind in ("pcg", "fgmres"):
        mats, prol, bds, rhs = _hierarchy(case, seed)
        precision = case.get("precision", "mixed")
        mg = MGPreconditioner(mats, prol, bds, [None] + [JacobiSmoother(2, 2 / 3)] * (len(mats) - 1), cycles=1,
                              use_fmg=False, precision=precision)
        solver = IterativeSolver()
        start = torch.zeros(len(rhs), dtype=torch.float64, device="cuda")
        state = {"kind": kind, "A": mats[-1], "b": torch.tensor(rhs, device="cuda"), "start": start,
                 "solver": solver, "tol": 1e-8 * float(np.linalg.norm(rhs)), "keep": (mats, prol, mg)}
        if kind == "pcg":
            start[0] = 1.0
            solver.precision = GRID_PRECISION[precision]
            state["M"] = mg
        else:
            H, W, dof = pixel_map(_space(1, case["coarse"] << (case["levels"] - 1)))
            net = LearnedSmoother(N.default_context(), weights=np.load(WEIGHTS))
            state["M"] = MGCNNPreconditioner(mg, net, mats[-1], H, W, dof, bds[-1])
        return state
    if kind == "mgapply":
        mats, prol, bds, rhs = _hierarchy(case, seed)
        mg = MGPreconditioner(mats, prol, bds, [None] + [JacobiSmoother(2, 2 / 3)] * (len(mats) - 1))
        return {"kind": kind, "M": mg, "v": rhs, "keep": (mats, prol)}
    if kind == "cnngrad":
        x, t, w = _images(case, seed)
        return {"kind": kind, "net": LearnedSmoother(N.default_context(), weights=w), "x": x, "t": t}
    if kind == "heat":
        cells, dts, u0 = _heat_inputs(case, seed)
        K, M, packed = [], [], []
        for c, dt, u in zip(cells, dts, u0):
            sp = _space(1, c)
            K.append(assemble_device(sp, dt, 1.0, dirichlet=False)[0])
            M.append(assemble_device(sp, 0.0, 1.0, dirichlet=False)[0])
            v = np.empty(sp.n)
            v[sp.node_of_grid] = u.numpy().reshape(-1)
            packed.append(v)
        return {"kind": kind, "batch": BatchedParabolicIntegrator(K, M), "u0": np.concatenate(packed),
                "steps": case["steps"]}
    if kind == "stokes":
        prob = stokes_problem(case["coarse"] << (case["levels"] - 1), case["coarse"], seed=seed & 0xFFFF,
                              pin_pressure=False)
        kw = {} if case["smoother"] == "schwarz" else {"smoother": "jacobi", "runs": 2, "omega": 0.6}
        return {"kind": kind, "S": StokesSolver(N.default_context(), prob, **kw),
                "tol": 1e-8 * float(np.linalg.norm(prob.system.rhs))}
    if kind == "dense":
        a, b = _dense_inputs(case["n"], seed)
        return {"kind": kind, "D": DenseMatrix(a), "b": b}
    sp, sc = _space(1, case["cells"]), _space(1, case["cells"] // 2)
    A, _, _, _ = assemble_device(sp, 1.0, 0.0, grad_coef_cells=_kappa_cells(case["cells"], seed))
    return {"kind": kind, "A": A, "P": DeviceMatrix(sp.n, sc.n, *_prolongation(1, sc.cx))}


def run(state):
    kind = state["kind"]
    if kind in ("cg", "pcg", "fgmres"):
        x = state["start"].clone()
        if kind == "cg":
            return state["solver"].solve_device(N.CG, state["A"], None, state["b"], x, state["tol"])
        if kind == "pcg":
            return state["solver"].solve_device(N.PCG, state["A"], state["M"], state["b"], x, state["tol"])
        return state["solver"].solve_device(N.FGMRES, state["A"], state["M"], state["b"], x, state["tol"], restart=30)
    if kind == "mgapply":
        return state["M"].mvMul(state["v"])
    if kind == "cnngrad":
        loss, grad = state["net"].loss_and_grad(state["x"], state["t"])
        return {"loss": loss, "grad": grad}
    if kind == "heat":
        return state["batch"].timeSteps(state["u0"], state["steps"])
    if kind == "stokes":
        x, _ = state["S"].solve(state["tol"])
        return x
    if kind == "dense":
        return state["D"].solve(state["b"])
    ptr, col, val = state["A"].galerkin(state["P"]).csr()
    return {"ptr": ptr, "col": col, "val": val}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _nnz(p, nodes):
    return (3 * nodes) ** 2 if p == 1 else (4 * nodes) ** 2


def work(case):
    """Each input read once, each output written once; one product per solve."""
    kind = case["kind"]
    if kind in ("cg", "pcg", "fgmres", "mgapply"):
        p = case.get("p", 1)
        cells = case["cells"] if kind == "cg" else case["coarse"] << (case["levels"] - 1)
        nodes = p * cells + 1
        nnz, n = _nnz(p, nodes), nodes * nodes
        flops = 2.0 * nnz
        if kind == "fgmres":
            flops += 2.0 * 37440 * n
        return {"bytes": 12.0 * nnz + 16.0 * n, "flops": flops}
    if kind == "cnngrad":
        px = case["batch"] * case["height"] * case["width"]
        return {"bytes": 8.0 * px + 8.0 * 37440, "flops": 6.0 * 37440 * px}
    if kind == "heat":
        cells, _, _ = _heat_inputs({**case}, 0)
        n = float(sum((c + 1) ** 2 for c in cells))
        return {"bytes": n * (2 * 9 * 12 + 16), "flops": n * 2 * 9 * 2 * case["steps"]}
    if kind == "stokes":
        c = case["coarse"] << (case["levels"] - 1)
        n = 2 * (2 * c + 1) ** 2 + (c + 1) ** 2
        return {"bytes": 12.0 * 34 * n + 16.0 * n, "flops": 2.0 * 34 * n}
    if kind == "dense":
        n = float(case["n"])
        return {"bytes": 8 * n * n + 16 * n, "flops": 2 * n ** 3 / 3}
    n = (case["cells"] + 1.0) ** 2
    return {"bytes": 12 * n * (9 + 2.25) + 12 * n * 9 / 4, "flops": 2 * n * 9 * 2.25 * 2}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
_GP = 0.5 * (np.polynomial.legendre.leggauss(5)[0] + 1)
_GW = 0.5 * np.polynomial.legendre.leggauss(5)[1]


def _line_elements(p, h):
    """1-D stiffness and mass matrices of one cell, equidistant Lagrange nodes."""
    nodes = np.arange(p + 1) / p
    co = np.linalg.inv(np.vander(nodes, p + 1, increasing=True))          # column i: coefficients of function i
    v = np.vander(_GP, p + 1, increasing=True) @ co
    d = np.stack([k * _GP ** max(k - 1, 0) for k in range(p + 1)], 1) @ co
    return (d.T * _GW) @ d / h, (v.T * _GW) @ v * h


def _line_matrices(p, cells):
    k, m = _line_elements(p, 1.0 / cells)
    n = p * cells + 1
    K, M = np.zeros((n, n)), np.zeros((n, n))
    for c in range(cells):
        K[c * p:c * p + p + 1, c * p:c * p + p + 1] += k
        M[c * p:c * p + p + 1, c * p:c * p + p + 1] += m
    return torch.tensor(K, device="cuda"), torch.tensor(M, device="cuda")


def _numbering(p, cells):
    """Unknown of every grid node (x-major): first appearance over cells (y fastest), local x fastest."""
    n = p * cells + 1
    i = np.arange(cells)
    loc = np.arange((p + 1) ** 2)
    gx = (i[:, None, None] * p + loc % (p + 1))
    gy = (i[None, :, None] * p + loc // (p + 1))
    visits = (gx * n + gy).reshape(-1)
    uniq, first = np.unique(visits, return_index=True)
    num = np.empty(n * n, dtype=np.int64)
    num[uniq[np.argsort(first, kind="stable")]] = np.arange(uniq.size)
    return num


def _grid_matrix(p, cells, kappa, mass):
    """CSR matrix on the node grid (x-major), zero Dirichlet rows and columns with a unit diagonal."""
    n = p * cells + 1
    k, m = _line_elements(p, 1.0 / cells)
    loc = np.arange((p + 1) ** 2)
    ax, ay = loc % (p + 1), loc // (p + 1)
    stiff = k[ax][:, ax] * m[ay][:, ay] + m[ax][:, ax] * k[ay][:, ay]
    massm = m[ax][:, ax] * m[ay][:, ay]
    i = np.arange(cells)
    nodes = ((i[:, None, None] * p + ax) * n + (i[None, :, None] * p + ay)).reshape(-1, loc.size)
    nodes = torch.tensor(nodes, device="cuda")
    kc = torch.ones(cells * cells, dtype=torch.float64, device="cuda") if kappa is None else \
        torch.tensor(kappa.reshape(-1), device="cuda")
    vals = kc[:, None, None] * torch.tensor(stiff, device="cuda") + mass * torch.tensor(massm, device="cuda")
    g = torch.arange(n, device="cuda")
    edge = (g == 0) | (g == n - 1)
    bd = (edge[:, None] | edge[None, :]).reshape(-1)
    r = nodes[:, :, None].expand_as(vals).reshape(-1)
    c = nodes[:, None, :].expand_as(vals).reshape(-1)
    keep = ~(bd[r] | bd[c])
    bi = bd.nonzero()[:, 0]
    r, c = torch.cat([r[keep], bi]), torch.cat([c[keep], bi])
    v = torch.cat([vals.reshape(-1)[keep], torch.ones(bi.numel(), dtype=torch.float64, device="cuda")])
    A = torch.sparse_coo_tensor(torch.stack([r, c]), v, (n * n, n * n)).coalesce()
    return A.to_sparse_csr(), bd


def _jacobi_pcg(A, b, rtol, maxit=60000):
    n = b.numel()
    crow, col, val = A.crow_indices(), A.col_indices(), A.values()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), crow.diff())
    d = torch.zeros_like(b)
    d[row[row == col]] = val[row == col]
    x = torch.zeros_like(b)
    for _ in range(3):                                   # restarted on the true residual
        r = b - A @ x
        z = r / d
        p = z.clone()
        rz = r @ z
        for it in range(maxit):
            q = A @ p
            alpha = rz / (p @ q)
            x += alpha * p
            r -= alpha * q
            z = r / d
            new = r @ z
            p = z + (new / rz) * p
            rz = new
            if it % 50 == 0 and float(r.norm()) <= rtol * float(b.norm()):
                break
    return x


def _to_dofs(grid, p, cells):
    out = np.empty(grid.numel())
    out[_numbering(p, cells)] = grid.cpu().numpy()
    return out


def _interp_1d(p, c):
    """Dense nodal interpolation from c to 2c cells."""
    nf = 2 * p * c + 1
    nodes = np.arange(p + 1) / p
    co = np.linalg.inv(np.vander(nodes, p + 1, increasing=True))
    P = np.zeros((nf, p * c + 1))
    for f in range(nf):
        k = min(f // (2 * p), c - 1)
        t = f / (2.0 * p) - k
        P[f, k * p:k * p + p + 1] += np.vander([t], p + 1, increasing=True)[0] @ co
    P[np.abs(P) < 1e-14] = 0
    return torch.tensor(P, device="cuda")


def _exact_mgapply(case, seed):
    p, cells, _, mass, load = _problem(case, seed)
    levels = case["levels"]
    A, bd = zip(*[_grid_matrix(p, case["coarse"] << l, None, mass) for l in range(levels)])
    P = [_interp_1d(p, case["coarse"] << l) for l in range(levels - 1)]
    dense0 = A[0].to_dense()
    idx = [torch.arange(a.shape[0], device="cuda") for a in A]
    diag = []
    for a, i in zip(A, idx):
        row = torch.repeat_interleave(i, a.crow_indices().diff())
        sel = row == a.col_indices()
        d = torch.zeros(a.shape[0], dtype=torch.float64, device="cuda")
        d[row[sel]] = a.values()[sel]
        diag.append(d)

    def up(l, v):
        n = P[l].shape[1]
        return (P[l] @ v.reshape(n, n) @ P[l].T).reshape(-1)

    def down(l, v):
        n = P[l].shape[0]
        return (P[l].T @ v.reshape(n, n) @ P[l]).reshape(-1).masked_fill(bd[l], 0)

    def smooth(l, x, b):
        for _ in range(2):
            x = x + (2 / 3) * (b - A[l] @ x) / diag[l]
        return x

    def cycle(l, x, b):
        if l == 0:
            return torch.linalg.solve(dense0, b)
        x = smooth(l, x, b)
        rc = down(l - 1, b - A[l] @ x)
        x = x + up(l - 1, cycle(l - 1, torch.zeros_like(rc), rc)).masked_fill(bd[l], 0)
        return smooth(l, x, b)

    v = torch.tensor(load.reshape(-1), device="cuda")
    first = v * bd[-1]
    defect = v - A[-1] @ first
    rhs = [defect]
    for l in range(levels - 2, -1, -1):
        rhs.insert(0, down(l, rhs[0]))
    x = torch.zeros_like(rhs[0])
    for l in range(levels - 1):
        x = up(l, cycle(l, x, rhs[l]))
    for _ in range(3):
        x = cycle(levels - 1, x, defect)
    return _to_dofs(x + first, p, cells)


def _exact_cnngrad(case, seed):
    x, t, flat = _images(case, seed)
    ws, o = [], 0
    for s in SHAPES:
        n = int(np.prod(s))
        ws.append(torch.tensor(flat[o:o + n].reshape(s), dtype=torch.float64, device="cuda", requires_grad=True))
        o += n
    conv = lambda v, w: torch.nn.functional.conv2d(v, w, padding=1)       # noqa: E731
    with torch.backends.cudnn.flags(enabled=False):
        h1 = conv(x[:, None].double(), ws[0]).relu()
        h3 = (h1 + conv(conv(h1, ws[1]).relu(), ws[2])).relu()
        h5 = (h3 + conv(conv(h3, ws[3]).relu(), ws[4])).relu()
        loss = ((conv(h5, ws[5])[:, 0] - t.double()) ** 2).mean()
        grads = torch.autograd.grad(loss, ws)
    return {"loss": float(loss), "grad": torch.cat([g.reshape(-1) for g in grads]).cpu().numpy()}


def _exact_heat(case, seed):
    cells, dts, u0 = _heat_inputs(case, seed)
    out, modes = [], {}
    for c, dt, u in zip(cells, dts, u0):
        if c not in modes:
            K, M = _line_matrices(1, c)
            Li = torch.linalg.inv(torch.linalg.cholesky(M))
            lam, Q = torch.linalg.eigh(Li @ K @ Li.T)
            V = Li.T @ Q                                  # V^T M V = I
            modes[c] = (lam, V, V.T @ M)
        lam, V, VM = modes[c]
        w = VM @ u.cuda() @ VM.T
        w = w / (1 + dt * (lam[:, None] + lam[None, :])) ** case["steps"]
        out.append(_to_dofs((V @ w @ V.T).reshape(-1), 1, c))
    return np.concatenate(out)


def _exact_stokes(case, seed):
    cells = case["coarse"] << (case["levels"] - 1)
    prob = stokes_problem(cells, cells, seed=seed & 0xFFFF, pin_pressure=True).system    # the COO triples and rhs
    n = prob.n
    A = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    idx = torch.tensor(prob.rows, device="cuda").long() * n + torch.tensor(prob.cols, device="cuda").long()
    A.index_add_(0, idx, torch.tensor(prob.vals, device="cuda"))
    x = torch.linalg.solve(A.view(n, n), torch.tensor(prob.rhs, device="cuda"))
    x[prob.nv:] -= x[prob.nv].clone()
    return x.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cg", "pcg", "fgmres"):
        if kind == "cg":
            p, cells, kappa, mass, load = 1, case["cells"], None, 5.0, _load_grid(case["cells"] + 1, seed, 4)
        else:
            p, cells, kappa, mass, load = _problem(case, seed)
        b = torch.tensor(load, device="cuda")
        if kappa is None:
            # constant coefficients: diagonalised direction by direction
            K, M = (m[1:-1, 1:-1] for m in _line_matrices(p, cells))
            Li = torch.linalg.inv(torch.linalg.cholesky(M))
            lam, Q = torch.linalg.eigh(Li @ K @ Li.T)
            V = Li.T @ Q
            w = (V.T @ b[1:-1, 1:-1] @ V) / (lam[:, None] + lam[None, :] + mass)
            x = torch.zeros_like(b)
            x[1:-1, 1:-1] = V @ w @ V.T
            x = x.reshape(-1)
        else:
            A, _ = _grid_matrix(p, cells, kappa[-1], mass)
            x = _jacobi_pcg(A, b.reshape(-1), 1e-13)
        return torch.tensor(_to_dofs(x, p, cells), device="cuda")
    if kind == "mgapply":
        return _exact_mgapply(case, seed)
    if kind == "cnngrad":
        return _exact_cnngrad(case, seed)
    if kind == "heat":
        return _exact_heat(case, seed)
    if kind == "stokes":
        return _exact_stokes(case, seed) if case["coarse"] << (case["levels"] - 1) <= 64 else None
    if kind == "dense":
        a, b = _dense_inputs(case["n"], seed)
        return torch.linalg.solve(torch.tensor(a, device="cuda"), torch.tensor(b, device="cuda")).cpu().numpy()
    cells = case["cells"]
    A, _ = _grid_matrix(1, cells, _kappa_cells(cells, seed), 0.0)
    num = torch.tensor(_numbering(1, cells), device="cuda")
    numc = torch.tensor(_numbering(1, cells // 2), device="cuda")
    P1 = _interp_1d(1, cells // 2)
    fx, cx = P1.nonzero(as_tuple=True)
    w = P1[fx, cx]
    n, nc = cells + 1, cells // 2 + 1
    rows = num[(fx[:, None] * n + fx[None, :]).reshape(-1)]
    cols = numc[(cx[:, None] * nc + cx[None, :]).reshape(-1)]
    P = torch.sparse_coo_tensor(torch.stack([rows, cols]), (w[:, None] * w[None, :]).reshape(-1),
                                (n * n, nc * nc)).coalesce()
    Ac = A.to_sparse_coo().coalesce()
    Ad = torch.sparse_coo_tensor(num[Ac.indices()], Ac.values(), Ac.shape).coalesce()
    C = torch.sparse.mm(torch.sparse.mm(P.t().coalesce(), Ad).coalesce(), P).coalesce()
    return {"ptr": None, "col": None, "val": C.values()[C.values() != 0].cpu().numpy()}
