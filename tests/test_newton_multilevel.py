"""BiCGStab with the multilevel cycle on scalar Jacobians: at the smallest
systems it is taken for (625 DoFs: one block; 729 and more: the grid), P1 and
P2, both diffusion forms, elimination and penalty rows, an initial guess, and a
Jacobian that it gives up on (the Jacobi iteration's answer then).

Tolerance: the residual is at most 1e-12 of b, the condition numbers of these
Jacobians are below 1e5: 1e-7 of the solution is the bound; what is asked is
1e-8, and 1e-11 (ten times the residual asked for) of the residual itself."""
import numpy as np
import pytest


def _system(G, ctx, order, n, form, amp, mode=None):
    from grmp_gb300 import fespace as F
    g = G.grid_unitsquare(n)
    S = F.FESpace(F.H1P1(1) if order == 1 else F.H1P2(1, 2), g)
    rng = np.random.default_rng(100 * order + n)
    ops = [G.LaplaceOperator(1.0), G.StructuralCoupling()]
    A = G.FEMatrix(ctx, S, ops)
    b, u, x = (G.FEVector(ctx, S) for _ in range(3))
    u.upload(amp * rng.standard_normal(S.ndofs))
    G.assemble(A, ops, G.FP64)
    b.upload(rng.standard_normal(S.ndofs))
    G.assemble_nonlinear(A, b, u, G.NonlinearForm(form, kappa=1.0, beta=1.0), G.FP64, add=True)
    G.apply_dirichlet(A, b, S.boundary_dofs(), None, mode if mode is not None else G.DIRICHLET_ELIMINATE)
    return A, b, x, S


@pytest.mark.gpu
@pytest.mark.parametrize("order,n", [(2, 12), (1, 26), (2, 13), (2, 20), (1, 41)])
@pytest.mark.parametrize("form", ["diffusion", "grad_diffusion"])
def test_solution(G, ctx, order, n, form):
    import scipy.sparse.linalg as spla
    A, b, x, S = _system(G, ctx, order, n, form, 0.1)
    solver = G.GB300PCG(mode="bicgstab", reltol=1e-12, abstol=0.0)
    st = solver.solve(A, b, x)
    assert st["spmv_config"] >= 90000
    M = A.download(G.FP64).tocsc()
    bh = b.entries
    assert np.linalg.norm(bh - M @ x.entries) <= 1e-11 * np.linalg.norm(bh)
    xr = spla.spsolve(M, bh)
    assert np.linalg.norm(x.entries - xr) <= 1e-8 * np.linalg.norm(xr)
    x.upload(xr + 1e-3 * np.random.default_rng(1).standard_normal(S.ndofs))
    st = G.GB300PCG(mode="bicgstab", reltol=1e-12, abstol=0.0, use_initial_guess=True).solve(A, b, x)
    assert np.linalg.norm(bh - M @ x.entries) <= 1e-11 * np.linalg.norm(bh)


@pytest.mark.gpu
def test_penalty_rows(G, ctx):
    A, b, x, S = _system(G, ctx, 2, 20, "diffusion", 0.1, G.DIRICHLET_PENALTY)
    G.GB300PCG(mode="bicgstab", reltol=1e-12, abstol=0.0).solve(A, b, x)
    free = np.setdiff1d(np.arange(S.ndofs), S.boundary_dofs())
    M, bh = A.download(G.FP64).tocsr(), b.entries
    assert np.linalg.norm((bh - M @ x.entries)[free]) <= 1e-11 * np.linalg.norm(bh[free])


@pytest.mark.gpu
def test_gives_up_and_leaves_the_jacobi_iterate(G, ctx):
    """Three iterations do not converge: the Jacobi iteration then starts from
    the same x, and x is its third iterate (compared with the same recurrence
    in NumPy: three steps of FP64 arithmetic, 1e-10)."""
    A, b, x, S = _system(G, ctx, 2, 20, "diffusion", 0.1)
    M, r = A.download(G.FP64).tocsr(), b.entries
    x0 = np.random.default_rng(2).standard_normal(S.ndofs)
    x.upload(x0)
    with pytest.raises(G.GrmpError):
        G.GB300PCG(mode="bicgstab", reltol=1e-12, abstol=0.0, maxiter=3, use_initial_guess=True).solve(A, b, x)
    d = M.diagonal()
    xr, r = x0.copy(), r - M @ x0
    rh, p, v, rho, alpha, omega = r.copy(), 0 * r, 0 * r, r @ r, 1.0, 1.0
    beta = 0.0
    for _ in range(3):
        p = r + beta * (p - omega * v)
        v = M @ (p / d)
        alpha = rho / (rh @ v)
        s = r - alpha * v
        t = M @ (s / d)
        omega = (t @ s) / (t @ t)
        xr = xr + alpha * p / d + omega * s / d
        r = s - omega * t
        rho, old = rh @ r, rho
        beta = rho / old * alpha / omega
    assert np.linalg.norm(x.entries - xr) <= 1e-10 * np.linalg.norm(xr)
