"""Batched Stokes direct solver: how a block's threads split into groups that
factor small fronts side by side depends on the batch's largest front (one,
two or four groups of whole warps).  Batches whose largest square gives fronts
below, between and above the rule's edges, against the oracle's sparse-direct
sweeps."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [10, 20, 28, 36, 41, 56, 68])
def test_direct_batch_over_front_sizes(G, O, ctx, n):
    """nu = 1, lambda = 1e4: cond ~ lambda n^2, so the bound is the cap of the
    conditioning bound that the other batch tests use, 1e-8."""
    from grmp_gb300 import stokes as S
    prob = S.make_batch(sizes=np.array([n, 7]), nus=np.array([1.0, 1.0]), seed=5)
    sysd = S.StokesBatchSystem(ctx, prob, mixed=False, direct=True)
    sysd.assemble()
    sysd.solve(sweeps=2, reltol=1e-13)
    u, p = sysd.velocity(), sysd.pressure()
    for k, g in enumerate(prob.mesh.parts):
        uo, po, _ = O.stokes_iterated_penalty(g, 1.0, prob.lam, prob.terms[k], sweeps=2)
        r0, r1 = prob.V.row_offsets[k], prob.V.row_offsets[k + 1]
        c0, c1 = prob.mesh.cell_offsets[k], prob.mesh.cell_offsets[k + 1]
        assert np.linalg.norm(u[r0:r1] - uo) <= 1e-8 * np.linalg.norm(uo)
        assert np.linalg.norm(p[c0:c1] - po) <= 1e-8 * np.linalg.norm(po)
