"""Face matrices in chunks.

3D P2 with 193,750 faces needs two chunks of face matrices (a chunk holds
512 MiB, 167,772 faces of this element): u^T J u must be the sum of the jump
integrals of u over the faces, which another kernel computes face by face.
Tolerance: both are sums of non-negative face terms with relative errors of
some hundred roundings, u^T J u of entries with cancelling signs (at most the
20 functions of a face): 20 x 100 x 2^-53 = 2e-13, taken ten times."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 25])
def test_quadratic_form_is_the_jump_integral(G, ctx, n):
    from grmp_gb300 import fespace as F
    g = G.grid_unitcube_kuhn(n)
    S = F.FESpace(F.H1P2(1, 3), g)
    op = G.BilinearForm([G.Jump(G.Gradient), G.Jump(G.Gradient)], G.FaceVolumePower(1.0), AT=G.ON_IFACES, factor=1.0)
    A = G.FEMatrix(ctx, S, [op])
    G.assemble(A, [op], G.FP64)
    u, y = G.FEVector(ctx, S), G.FEVector(ctx, S)
    uh = np.random.default_rng(n).standard_normal(S.ndofs)
    u.upload(uh)
    G.spmv(A, u, y, G.FP64)
    ref = G.FaceJumpIntegrator(normal=False, power=1.0, factor=1.0).evaluate_faces(u).sum()
    assert abs(uh @ y.entries - ref) <= 2e-12 * ref
