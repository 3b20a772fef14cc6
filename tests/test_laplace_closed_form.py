"""Assembly of a single Laplace term in closed form against the contraction
with reference tensors, which a second term of factor zero selects: P1 and P2,
2D and 3D, scalar and vector spaces, distorted cells of both orientations,
jumping cell coefficients, every precision.

Tolerance: an entry is a sum of at most 24 cells' contributions of some 20
roundings each, 24 x 20 x 2^-53 = 5e-14 of the largest entry in FP64 and 3e-5
in FP32; the contributions of a cell differ in size by less than a factor 20
from its largest, so 1e-12 and 6e-4 are asked."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("dim,order,nc,n", [(2, 1, 1, 1), (2, 1, 1, 12), (2, 2, 1, 1), (2, 2, 1, 12), (2, 2, 2, 5),
                                            (2, 1, 2, 5), (3, 1, 1, 1), (3, 1, 1, 5), (3, 2, 1, 1), (3, 2, 1, 5)])
def test_matches_tensor_contraction(G, ctx, dim, order, nc, n):
    from grmp_gb300 import fespace as F
    from grmp_gb300 import mesh as M
    g0 = G.grid_unitsquare(n) if dim == 2 else G.grid_unitcube_kuhn(n)
    rng = np.random.default_rng(10 * dim + order + n)
    cells = np.array(g0.cells)
    cells[::3, :2] = cells[::3, 1::-1]   # every third cell the other way round
    g = M.SimplexMesh(np.array(g0.coords) + 0.2 / n * (rng.random(g0.coords.shape) - 0.5), cells)
    S = F.FESpace(F.H1P1(nc) if order == 1 else F.H1P2(nc, dim), g)
    lap = G.BilinearForm([G.Gradient, G.Gradient], G.CellCoefficient(np.exp(rng.standard_normal(g.ncells))),
                         APT=G.APT_SymmetricBilinearForm)
    one, two = [lap], [lap, G.ReactionOperator(0.0)]
    A, B = G.FEMatrix(ctx, S, [lap, G.StructuralCoupling()]), G.FEMatrix(ctx, S, [lap, G.StructuralCoupling()])
    G.assemble(A, one, G.FP64_FP32)
    G.assemble(B, two, G.FP64_FP32)
    a, b = A.download(G.FP64).data, B.download(G.FP64).data
    assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
    a32, b32 = A.download(G.FP32).data, B.download(G.FP32).data
    assert np.max(np.abs(a32 - b32)) <= 6e-4 * np.max(np.abs(b32))
    G.assemble(A, one, G.FP64)
    G.assemble(A, one, G.FP32)
    assert np.array_equal(A.download(G.FP64).data, a) and np.array_equal(A.download(G.FP32).data, a32)
