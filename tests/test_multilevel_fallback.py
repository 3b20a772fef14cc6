"""Multilevel conjugate gradients on matrices that the cycle does not suit: jumps
of 1e5 and 1e6 in the coefficient and a thin strip fixed at one end, where the
FP32 recurrence loses its conjugacy and the FP64 cycle has to take over, and
solves that the caller's maxiter ends, which the Jacobi iteration goes on with.

Tolerance: the FP64 recurrence stops at the tolerance asked for; its residual
departs from b - A x by rounding of iterates times the matrix's condition, ten
times the tolerance is allowed.  Iterations: FP64 needs some hundreds (condition
about 1e7 to 1e10, aggregates inside one material), a solve that fails all
20,000."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(G, ctx, kind, n, order=1):
    from grmp_gb300 import fespace as F
    from grmp_gb300 import mesh as M
    g = G.grid_unitsquare(n)
    X = np.array(g.coords)
    if kind == "strip":
        X[:, 1] *= 0.03
    g = M.SimplexMesh(X, np.array(g.cells))
    mid = X[np.array(g.cells)].mean(axis=1)
    S = F.FESpace(F.H1P1(1) if order == 1 else F.H1P2(1, 2), g)
    c = np.ones(g.ncells)
    fixed = S.boundary_dofs()
    if kind == "strip":
        fixed = np.flatnonzero(X[:, 0] < 1e-12).astype(np.int32)   # P1: DoFs are vertices
    else:
        f = np.floor(mid * 8).astype(int)
        c[(f.sum(axis=1) % 2 == 0) & np.all(mid * 8 - f > 0.25, axis=1)] = kind
    ops = [G.BilinearForm([G.Gradient, G.Gradient], G.CellCoefficient(c), APT=G.APT_SymmetricBilinearForm)]
    A = G.FEMatrix(ctx, S, ops)
    b, x = G.FEVector(ctx, S), G.FEVector(ctx, S)
    G.assemble(A, ops, G.FP64_FP32)
    b.upload(np.random.default_rng(2).standard_normal(S.ndofs))
    G.apply_dirichlet(A, b, fixed, None, G.DIRICHLET_ELIMINATE)
    return A, b, x, S


def _relres(G, A, b, x):
    bh = b.entries
    return np.linalg.norm(bh - A.download(G.FP64).tocsr() @ x.entries) / np.linalg.norm(bh)


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("kind,n,order,tol", [(1e5, 80, 1, 1e-8), (1e6, 80, 1, 1e-8), (1e6, 64, 2, 1e-8),
                                              (1e5, 24, 1, 1e-8), ("strip", 80, 1, 1e-4)])
def test_converges(G, ctx, kind, n, order, tol, mode):
    A, b, x, S = _problem(G, ctx, kind, n, order)
    st = G.GB300PCG(mode=mode, reltol=tol, abstol=0.0, maxiter=20000).solve(A, b, x)
    assert st["iterations"] <= 1000
    assert _relres(G, A, b, x) <= 10 * tol
    # from a start whose residual is larger than b
    x.upload(x.entries * (1 + 1e-3 * np.cos(np.arange(S.ndofs))))
    G.GB300PCG(mode=mode, reltol=tol, abstol=0.0, maxiter=20000, use_initial_guess=True).solve(A, b, x)
    assert _relres(G, A, b, x) <= 10 * tol


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("entry", ["solve", "noalloc"])
def test_maxiter_is_followed_by_the_jacobi_iteration(G, ctx, mode, entry):
    """Three iterations of the cycle and three of Jacobi-CG from where they led."""
    from grmp_gb300 import _lib as L
    if entry == "noalloc" and mode == "mixed":
        pytest.skip("FP64 only")
    A, b, x, S = _problem(G, ctx, 1.0, 40)
    solver = G.GB300PCG(mode=mode, reltol=1e-11, abstol=0.0)
    assert solver.solve(A, b, x)["spmv_config"] >= 90000   # the hierarchy is there
    sol = x.entries.copy()
    x.fill(0.0)
    solver.maxiter = 3
    if entry == "solve":
        st = solver.solve(A, b, x, raise_on_error=False)
        assert st["rc"] == st["status"] and st["spmv_config"] < 90000
        assert st["iterations"] == 3
        rc = st["rc"]
    else:
        p, s = solver.params(), L.SolveStats()
        rc = ctx.lib.grmp_solve_fp64_noalloc(A.h, b.h, x.h, ctypes.byref(p), ctypes.byref(s))
        assert s.iterations == 3 and s.spmv_config < 90000
    assert rc != 0
    # three cycles alone bring the error of this problem below a half of the solution
    assert np.linalg.norm(x.entries - sol) <= 0.5 * np.linalg.norm(sol)
