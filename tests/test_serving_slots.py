"""Requests of different sizes on four slots at once, many times over: launches
of the same kernels with different shared-memory sizes from several threads must
not disturb each other.  Every answer equals, bit for bit, the one that a server
with one slot gives."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_slots_do_not_disturb_each_other(G):
    from grmp_gb300 import fespace as F
    from grmp_gb300 import serve as SV
    rng = np.random.default_rng(7)
    reqs = []
    for dim, order, n in ((2, 1, 30), (2, 2, 12), (3, 1, 13), (3, 2, 6), (2, 2, 25), (3, 2, 4)):
        g = G.grid_unitsquare(n) if dim == 2 else G.grid_unitcube_kuhn(n)
        S = F.FESpace(F.H1P1(1) if order == 1 else F.H1P2(1, dim), g)
        reqs.append(SV.ServeRequest(dim, order, n, S, np.exp(rng.standard_normal(g.ncells)), 0.0, rng.standard_normal(4),
                                    rng.integers(1, 4, size=(4, dim)).astype(float), S.boundary_dofs(),
                                    mesh_key=SV.mesh_key(dim, n, order)))
    one, four = SV.Server(0, 8 << 30, 1), SV.Server(0, 8 << 30, 4)
    ref = []
    for r in reqs:
        one.wait(one.submit(r, "mixed", 1e-11), r.ndofs)
        rc, x, _ = one.wait(one.submit(r, "mixed", 1e-11), r.ndofs)
        assert rc == 0
        ref.append(x.copy())
    for _ in range(40):
        ids = [four.submit(r, "mixed", 1e-11) for r in reqs]
        for r, i, x0 in zip(reqs, ids, ref):
            rc, x, _ = four.wait(i, r.ndofs)
            assert rc == 0 and np.array_equal(x, x0)
