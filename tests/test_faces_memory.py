"""Face terms where memory is short: accepted with a few bytes of scratch, and
the same bits as with room for the face matrices (in one chunk and, 193,750
faces of 3D P2, in two)."""
import numpy as np
import pytest


def _values(G, ctx, dim, order, n, prec, budget_left=None):
    """Values of Laplace + gradient jumps; budget_left: bytes that the budget
    leaves when the matrix stands."""
    from grmp_gb300 import fespace as F
    g = G.grid_unitsquare(n) if dim == 2 else G.grid_unitcube_kuhn(n)
    S = F.FESpace(F.H1P1(1) if order == 1 else F.H1P2(1, dim), g)
    ops = [G.LaplaceOperator(1.0), G.BilinearForm([G.Jump(G.Gradient), G.Jump(G.Gradient)], G.FaceVolumePower(2.0),
                                                  AT=G.ON_IFACES, factor=0.3)]
    A = G.FEMatrix(ctx, S, ops)
    G.assemble(A, ops, prec)
    hold = None
    if budget_left is not None:
        class H:
            ndofs = (budget_left[0] - ctx.memory_in_use() - budget_left[1]) // 8
        hold = G.FEVector(ctx, H)
        G.assemble(A, ops, prec)
    used = ctx.memory_in_use()
    del hold
    return A.download(G.FP64).data, A.download(G.FP32).data if prec == G.FP64_FP32 else None, used


@pytest.mark.gpu
@pytest.mark.parametrize("dim,order,n", [(2, 1, 1), (2, 1, 37), (2, 2, 30), (3, 1, 9), (3, 2, 6), (3, 2, 25)])
def test_same_bits_with_little_memory(G, ctx, dim, order, n):
    v64, v32, _ = _values(G, ctx, dim, order, n, G.FP64_FP32)
    budget = 8 << 30
    left = 2000 if (dim, order) == (3, 2) else 600   # the cells' assembly takes 1,408 bytes of scratch there
    small = G.GB300Context(0, hbm_budget_bytes=budget)
    w64, w32, used = _values(G, small, dim, order, n, G.FP64_FP32, (budget, left))
    assert used > budget - left - 8
    assert np.array_equal(v64, w64) and np.array_equal(v32, w32)
