"""Direct solves of matrices with face terms, whose pattern couples DoFs across
the separators of the cells' graph: both modes on the gradient-jump stabilised
operator, 2D and 3D, P1 and P2, more DoFs than a leaf of the ordering holds.

Tolerance: the solver refines to a residual of 1e-12 of b, ten times that is
asked for; condition numbers are below 1e4 (at most 729 DoFs, and the jump term
adds a fourth-order part of the operator's own size): 1e-8 bounds the error."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["direct", "mixed_direct"])
@pytest.mark.parametrize("dim,order,n", [(2, 1, 7), (2, 1, 16), (2, 2, 4), (2, 2, 11), (3, 1, 4), (3, 1, 7), (3, 2, 2),
                                         (3, 2, 4)])
def test_stabilised_operator(G, ctx, dim, order, n, mode):
    import scipy.sparse.linalg as spla
    from grmp_gb300 import fespace as F
    g = G.grid_unitsquare(n) if dim == 2 else G.grid_unitcube_kuhn(n)
    S = F.FESpace(F.H1P1(1) if order == 1 else F.H1P2(1, dim), g)
    ops = [G.LaplaceOperator(1.0),
           G.BilinearForm([G.Jump(G.Gradient), G.Jump(G.Gradient)], G.FaceVolumePower(2.0), AT=G.ON_IFACES, factor=0.1)]
    A = G.FEMatrix(ctx, S, ops)
    b, x = G.FEVector(ctx, S), G.FEVector(ctx, S)
    G.assemble(A, ops, G.FP64)
    b.upload(np.random.default_rng(n).standard_normal(S.ndofs))
    G.apply_dirichlet(A, b, S.boundary_dofs(), None, G.DIRICHLET_ELIMINATE)
    G.GB300PCG(mode=mode, reltol=1e-12, abstol=0.0).solve(A, b, x)
    M, bh = A.download(G.FP64).tocsc(), b.entries
    assert np.linalg.norm(bh - M @ x.entries) <= 1e-11 * np.linalg.norm(bh)
    xr = spla.spsolve(M, bh)
    assert np.linalg.norm(x.entries - xr) <= 1e-8 * np.linalg.norm(xr)
