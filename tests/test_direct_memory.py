"""What a direct solve leaves allocated: the factor and its updates, not the
buffers of the large fronts, of which a factorisation takes as many as it can get.
The smallest budget that the solve runs in holds the factor, one buffer and the
vectors, so that much is the bound for what stays."""
import numpy as np
import pytest


def _solve(G, ctx, mode):
    from grmp_gb300 import fespace as F
    S = F.FESpace(F.H1P2(2, 2), G.grid_unitsquare(40))
    ops = [G.HookStiffnessOperator2D(1.0, 1e3)]
    A = G.FEMatrix(ctx, S, ops)
    b, x = G.FEVector(ctx, S), G.FEVector(ctx, S)
    G.assemble(A, ops, G.FP64)
    b.upload(np.random.default_rng(1).standard_normal(S.ndofs))
    G.apply_dirichlet(A, b, S.boundary_dofs(), None, G.DIRICHLET_ELIMINATE)
    G.GB300PCG(mode=mode, reltol=1e-12, abstol=0.0).solve(A, b, x)
    return ctx.memory_in_use(), x.entries.copy()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["direct", "mixed_direct"])
def test_the_front_buffers_are_given_back(G, mode):
    stays, ref = _solve(G, G.GB300Context(0), mode)
    lo, hi = 1 << 20, 1 << 30
    while hi - lo > 64 << 10:
        mid = (lo + hi) // 2
        try:
            _, x = _solve(G, G.GB300Context(0, hbm_budget_bytes=mid), mode)
            assert np.array_equal(x, ref)
            hi = mid
        except G.GrmpError as e:
            assert "BUDGET" in str(e)
            lo = mid
    assert stays <= hi
