"""Vertex level of the multilevel hierarchy on meshes whose cells cancel for the
unit coefficient: the diagonals of isosceles trapezoids have no P1 stiffness in
sum, but do couple when the coefficient varies from cell to cell.

Tolerance: the solver stops at a residual of 1e-11 of b, ten times that is asked
for.  Iterations: moving the vertices by a ten-thousandth of the mesh width
changes no angle by more than about 1e-4 and undoes every cancellation, so the
hierarchy of the trapezoids has to converge as that one does; a quarter more and
five iterations are allowed for the different aggregates."""
import numpy as np
import pytest


def trapezoids(G, n, height, shift, noise):
    """Unit square grid, rows of height `height`, every other vertex of every
    other row moved so that all quads are isosceles trapezoids."""
    from grmp_gb300 import mesh as M
    g = G.grid_unitsquare(n)
    X = np.array(g.coords)
    i, j = np.rint(X * n).astype(int).T
    inner = (i > 0) & (i < n)
    X[:, 0] += np.where((j % 2 == 1) & inner, np.where(i % 2 == 1, 1.0, -1.0) * shift / n, 0.0)
    X[:, 1] *= height
    X += noise / n * inner[:, None] * (np.random.default_rng(7).random(X.shape) - 0.5)
    return M.SimplexMesh(X, np.array(g.cells))


def _solve(G, ctx, n, height, shift, sigma, prec, noise):
    from grmp_gb300 import fespace as F
    g = trapezoids(G, n, height, shift, noise)
    S = F.FESpace(F.H1P2(1, 2), g)
    rng = np.random.default_rng(n)
    ops = [G.BilinearForm([G.Gradient, G.Gradient], G.CellCoefficient(np.exp(sigma * rng.standard_normal(g.ncells))),
                          APT=G.APT_SymmetricBilinearForm)]
    A = G.FEMatrix(ctx, S, ops)
    b, x = G.FEVector(ctx, S), G.FEVector(ctx, S)
    G.assemble(A, ops, G.FP64_FP32 if prec == "mixed" else G.FP64)
    b.upload(rng.standard_normal(S.ndofs))
    G.apply_dirichlet(A, b, S.boundary_dofs(), None, G.DIRICHLET_ELIMINATE)
    st = G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0, maxiter=3000).solve(A, b, x)
    assert st["spmv_config"] >= 90000
    M, bh = A.download(G.FP64).tocsr(), b.entries
    assert np.linalg.norm(bh - M @ x.entries) <= 1e-10 * np.linalg.norm(bh)
    return st["iterations"]


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("sigma", [1.0, 2.0])
@pytest.mark.parametrize("n,height,shift", [(16, 0.5, 0.2), (32, 0.4, 0.2), (33, 0.5, 0.3)])
def test_isosceles_trapezoids(G, ctx, n, height, shift, sigma, prec):
    its = _solve(G, ctx, n, height, shift, sigma, prec, 0.0)
    assert its <= 1.25 * _solve(G, ctx, n, height, shift, sigma, prec, 1e-4) + 5
