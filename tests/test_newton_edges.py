"""BiCGStab with the multilevel cycle at the edges of its size rule, both sides,
2D (from 200 rows) and 3D (from 500), P1 and P2.

Tolerance: the residual asked for is 1e-12 of b, ten times that is allowed;
condition numbers are below 1e4 at these sizes, 1e-8 of the solution."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("dim,order,n,multilevel", [(2, 1, 13, False), (2, 1, 14, True), (2, 2, 6, False), (2, 2, 7, True),
                                                    (3, 1, 6, False), (3, 1, 7, True), (3, 2, 3, False), (3, 2, 4, True)])
def test_size_rule(G, ctx, dim, order, n, multilevel):
    import scipy.sparse.linalg as spla
    from grmp_gb300 import fespace as F
    g = G.grid_unitsquare(n) if dim == 2 else G.grid_unitcube_kuhn(n)
    S = F.FESpace(F.H1P1(1) if order == 1 else F.H1P2(1, dim), g)
    rng = np.random.default_rng(n)
    ops = [G.LaplaceOperator(1.0), G.StructuralCoupling()]
    A = G.FEMatrix(ctx, S, ops)
    b, u, x = (G.FEVector(ctx, S) for _ in range(3))
    u.upload(0.1 * rng.standard_normal(S.ndofs))
    G.assemble(A, ops, G.FP64)
    b.upload(rng.standard_normal(S.ndofs))
    G.assemble_nonlinear(A, b, u, G.NonlinearForm("diffusion", kappa=1.0, beta=1.0), G.FP64, add=True)
    G.apply_dirichlet(A, b, S.boundary_dofs(), None, G.DIRICHLET_ELIMINATE)
    st = G.GB300PCG(mode="bicgstab", reltol=1e-12, abstol=0.0).solve(A, b, x)
    assert (st["spmv_config"] >= 90000) == multilevel
    M, bh = A.download(G.FP64).tocsc(), b.entries
    assert np.linalg.norm(bh - M @ x.entries) <= 1e-11 * np.linalg.norm(bh)
    xr = spla.spsolve(M, bh)
    assert np.linalg.norm(x.entries - xr) <= 1e-8 * np.linalg.norm(xr)
