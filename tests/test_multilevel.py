"""Multilevel preconditioned solves: the smallest systems of each kind that
take them (one block and the grid, vertex and aggregated first levels, block and
group forms of the products), Dirichlet rows by elimination and penalty, an
initial guess, general meshes, reaction-dominated and explicitly configured
solves, which keep the Jacobi iteration, and the entry that allocates nothing.

Tolerance: the solver stops at a residual of 1e-11 of b and ten times that is
asked for; the systems whose error is compared (below 8,000 rows) have condition
numbers below 1e5: 1e-8."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(G, ctx, dim, order, n, prec, reaction=0.0, seed=0, distort=0.0, dirichlet=True, mode=None):
    from grmp_gb300 import fespace as F
    from grmp_gb300 import mesh as M
    g = G.grid_unitsquare(n) if dim == 2 else G.grid_unitcube_kuhn(n)
    rng = np.random.default_rng(seed)
    if distort:
        X = np.array(g.coords)
        inner = np.all((X > 1e-9) & (X < 1 - 1e-9), axis=1)
        X[inner] += distort / n * (rng.random((inner.sum(), dim)) - 0.5)
        g = M.SimplexMesh(X, np.array(g.cells))
    S = F.FESpace(F.H1P1(1) if order == 1 else F.H1P2(1, dim), g)
    ops = [G.BilinearForm([G.Gradient, G.Gradient], G.CellCoefficient(np.exp(rng.standard_normal(g.ncells))),
                          APT=G.APT_SymmetricBilinearForm)]
    if reaction:
        ops.append(G.ReactionOperator(reaction))
    A = G.FEMatrix(ctx, S, ops)
    b, x = G.FEVector(ctx, S), G.FEVector(ctx, S)
    G.assemble(A, ops, G.FP64_FP32 if prec == "mixed" else G.FP64)
    b.upload(rng.standard_normal(S.ndofs))
    if dirichlet:
        G.apply_dirichlet(A, b, S.boundary_dofs(), None, mode if mode is not None else G.DIRICHLET_ELIMINATE)
    return A, b, x, S


def _check(G, A, b, x, rows=slice(None)):
    M, bh, xh = A.download(G.FP64).tocsr(), b.entries, x.entries
    r = (bh - M @ xh)[rows]
    assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(bh[rows])
    return M, bh, xh


@pytest.mark.parametrize("dim,order,n,prec", [
    # the smallest systems that take it
    (2, 1, 10, "mixed"), (2, 2, 5, "mixed"), (2, 1, 20, "fp64"), (2, 2, 10, "fp64"), (3, 1, 13, "mixed"),
    (3, 1, 12, "fp64"), (3, 2, 6, "mixed"), (3, 2, 5, "fp64"),
    # on both sides of one block / the grid
    (2, 1, 23, "fp64"), (2, 1, 24, "fp64"), (2, 2, 19, "mixed"), (2, 2, 20, "mixed"),
    # on both sides of multiplicative / additive smoothing of the fine level
    (3, 2, 21, "mixed"), (3, 2, 22, "mixed"), (3, 2, 21, "fp64"), (3, 2, 22, "fp64"), (2, 1, 631, "mixed"),
    (2, 1, 632, "mixed")])
def test_smallest_systems(G, ctx, dim, order, n, prec):
    import scipy.sparse.linalg as spla
    A, b, x, S = _system(G, ctx, dim, order, n, prec)
    st = G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0).solve(A, b, x)
    assert st["spmv_config"] >= 90000
    M, bh, xh = _check(G, A, b, x)
    if S.ndofs < 8000:
        xr = spla.spsolve(M.tocsc(), bh)
        assert np.linalg.norm(xh - xr) <= 1e-8 * np.linalg.norm(xr)
    again = xh.copy()
    x.fill(0.0)
    G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0).solve(A, b, x)
    assert np.array_equal(x.entries, again)
    x.upload(again * (1 + 1e-4 * np.cos(np.arange(S.ndofs))))
    G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0, use_initial_guess=True).solve(A, b, x)
    _check(G, A, b, x)


@pytest.mark.parametrize("dim,order,n,prec", [(2, 2, 30, "fp64"), (2, 1, 45, "mixed"), (3, 2, 9, "mixed")])
def test_distorted_mesh(G, ctx, dim, order, n, prec):
    A, b, x, S = _system(G, ctx, dim, order, n, prec, distort=0.4, seed=3)
    st = G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0).solve(A, b, x)
    assert st["spmv_config"] >= 90000
    _check(G, A, b, x)


def test_penalty_rows(G, ctx):
    A, b, x, S = _system(G, ctx, 2, 2, 20, "fp64", mode=G.DIRICHLET_PENALTY)
    G.GB300PCG(mode="fp64", reltol=1e-11, abstol=0.0).solve(A, b, x)
    _check(G, A, b, x, np.setdiff1d(np.arange(S.ndofs), S.boundary_dofs()))


def test_small_reaction_without_dirichlet_rows(G, ctx):
    """Natural boundary: nearly singular, the constant is in the bottom level."""
    A, b, x, S = _system(G, ctx, 2, 2, 20, "fp64", reaction=1.0, dirichlet=False)
    st = G.GB300PCG(mode="fp64", reltol=1e-11, abstol=0.0).solve(A, b, x)
    assert st["spmv_config"] >= 90000
    _check(G, A, b, x)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_what_keeps_the_jacobi_iteration(G, ctx, prec):
    A, b, x, S = _system(G, ctx, 2, 2, 20, prec, reaction=1e6)
    st = G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0).solve(A, b, x)
    assert st["spmv_config"] < 90000      # reaction dominated
    _check(G, A, b, x)
    A, b, x, S = _system(G, ctx, 2, 2, 20, prec)
    st = G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0, spmv_config=404).solve(A, b, x)
    assert st["spmv_config"] == 404       # asked for
    _check(G, A, b, x)
    A, b, x, S = _system(G, ctx, 2, 1, 9, prec)
    st = G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0).solve(A, b, x)
    assert st["spmv_config"] < 90000      # 100 rows
    _check(G, A, b, x)


def test_new_values_on_a_built_hierarchy(G, ctx):
    """The hierarchy's values follow the matrix; its patterns stay."""
    A, b, x, S = _system(G, ctx, 2, 2, 20, "fp64")
    solver = G.GB300PCG(mode="fp64", reltol=1e-11, abstol=0.0)
    solver.solve(A, b, x)
    rng = np.random.default_rng(8)
    op = [G.BilinearForm([G.Gradient, G.Gradient], G.CellCoefficient(np.exp(2 * rng.standard_normal(S.xgrid.ncells))),
                         APT=G.APT_SymmetricBilinearForm)]
    G.assemble(A, op, G.FP64)
    G.apply_dirichlet(A, b, S.boundary_dofs(), None, G.DIRICHLET_ELIMINATE)
    solver.solve(A, b, x)
    _check(G, A, b, x)


def test_not_converged_and_without_allocation(G, ctx):
    from grmp_gb300 import _lib as L
    A, b, x, S = _system(G, ctx, 2, 2, 20, "fp64")
    with pytest.raises(G.GrmpError):
        G.GB300PCG(mode="fp64", reltol=1e-11, abstol=0.0, maxiter=2).solve(A, b, x)
    solver = G.GB300PCG(mode="fp64", reltol=1e-11, abstol=0.0)
    solver.solve(A, b, x)
    ref = x.entries.copy()
    x.fill(0.0)
    used = ctx.memory_in_use()
    p, st = solver.params(), L.SolveStats()
    assert ctx.lib.grmp_solve_fp64_noalloc(A.h, b.h, x.h, ctypes.byref(p), ctypes.byref(st)) == 0
    assert ctx.memory_in_use() == used and np.array_equal(x.entries, ref)
