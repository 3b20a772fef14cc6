"""Reaction-dominated matrices keep the Jacobi iteration and pay neither the
analysis nor the memory of a hierarchy they never use; a bad diagonal is still
refused."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(G, ctx, n, order, reaction, prec, laplace=1.0):
    from grmp_gb300 import fespace as F
    S = F.FESpace(F.H1P1(1) if order == 1 else F.H1P2(1, 2), G.grid_unitsquare(n))
    ops = [G.LaplaceOperator(laplace), G.ReactionOperator(reaction)]
    A = G.FEMatrix(ctx, S, ops)
    b, x = G.FEVector(ctx, S), G.FEVector(ctx, S)
    G.assemble(A, ops, G.FP64_FP32 if prec == "mixed" else G.FP64)
    b.upload(np.random.default_rng(n).standard_normal(S.ndofs))
    return A, b, x, S, ops


@pytest.mark.parametrize("prec", ["fp64", "mixed", "bicgstab"])
@pytest.mark.parametrize("order,n", [(1, 40), (2, 30)])
def test_no_memory_where_it_is_not_used(G, ctx, order, n, prec):
    """What the solve leaves allocated is what the Jacobi configuration leaves
    (the solver's workspace)."""
    left = []
    for cfg in (404, 0):
        A, b, x, S, ops = _system(G, ctx, n, order, 1e7, prec)
        before = ctx.memory_in_use()
        st = G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0, spmv_config=cfg).solve(A, b, x)
        assert st["spmv_config"] < 90000
        left.append(ctx.memory_in_use() - before)
        r = b.entries - A.download(G.FP64).tocsr() @ x.entries
        assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(b.entries)
    assert left[1] <= left[0]


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_hierarchy_for_later_values(G, ctx, prec):
    """Reaction dominated at first, elliptic at the next assembly: the cycle then."""
    A, b, x, S, ops = _system(G, ctx, 30, 2, 1e7, prec)
    solver = G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0)
    assert solver.solve(A, b, x)["spmv_config"] < 90000
    G.assemble(A, [G.LaplaceOperator(1.0), G.ReactionOperator(1.0)], G.FP64_FP32 if prec == "mixed" else G.FP64)
    assert solver.solve(A, b, x)["spmv_config"] >= 90000
    r = b.entries - A.download(G.FP64).tocsr() @ x.entries
    assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(b.entries)


@pytest.mark.parametrize("prec", ["fp64", "mixed", "bicgstab"])
@pytest.mark.parametrize("reaction", [0.0, 1e7])
def test_bad_diagonal_is_refused(G, ctx, prec, reaction):
    A, b, x, S, ops = _system(G, ctx, 30, 2, -reaction, prec, laplace=-1.0)
    with pytest.raises(G.GrmpError, match="diagonal"):
        G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0).solve(A, b, x)


@pytest.mark.parametrize("prec", ["fp64", "mixed", "bicgstab"])
def test_looked_at_once_per_values(G, ctx, prec):
    """A repeated solve of the same values launches one kernel less; assembly and
    Dirichlet rows make new values."""
    A, b, x, S, ops = _system(G, ctx, 30, 2, 1e7, prec)

    def launches():
        n0, n1 = ctypes.c_uint64(), ctypes.c_uint64()
        ctx.check(ctx.lib.grmp_context_launches(ctx.h, ctypes.byref(n0)))
        G.GB300PCG(mode=prec, reltol=1e-11, abstol=0.0, spmv_config=-1).solve(A, b, x)
        ctx.check(ctx.lib.grmp_context_launches(ctx.h, ctypes.byref(n1)))
        return n1.value - n0.value
    launches()   # builds what the Jacobi solver keeps
    again = launches()
    G.assemble(A, ops, G.FP64_FP32 if prec == "mixed" else G.FP64)
    assert launches() == again + 1 and launches() == again
    G.apply_dirichlet(A, b, S.boundary_dofs(), None, G.DIRICHLET_ELIMINATE)
    assert launches() == again + 1 and launches() == again
