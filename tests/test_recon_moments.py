"""Reconstructed Bernardi-Raugel right-hand sides from the data's vertex
moments: exponents that are decoded to integers (0..8) and those that go
through pow (9, 2.5), RT0 and BDM1, on cell counts off the block size, against
the oracle's evaluation of every reconstructed function.

Tolerance: both sides sum the same quadrature points in FP64, some 100
operations an entry, 100 x 2^-53 = 1.1e-14 of the sum of magnitudes; the
entries cancel at most to their hundredth part: 1e-12 of the largest."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("dim,n", [(2, 1), (2, 9), (3, 1), (3, 3)])
@pytest.mark.parametrize("recon", [1, 2])
def test_rhs_exponents(G, O, ctx, dim, n, recon):
    from grmp_gb300 import api
    from grmp_gb300 import fespace as F
    g = G.grid_unitsquare(n) if dim == 2 else G.grid_unitcube_kuhn(n)
    FES = F.FESpace(F.H1BR(dim), g)
    rng = np.random.default_rng(10 * dim + n)
    terms = np.array([(c, rng.standard_normal(), *np.roll([e, 1.0, 2.0][:dim] + [0.0] * (3 - dim), 0))
                      for c in range(dim) for e in (0.0, 1.0, 2.0, 3.0, 8.0, 9.0, 2.5)])
    op = {1: api.ReconstructionIdentity, 2: api.ReconstructionIdentityBDM1}[recon]
    _, ref, _, _, _ = O.br_stokes_system(g, 1.0, 0.0, terms, bonus_quadorder=1, recon=recon)
    b = api.FEVector(ctx, FES)
    b.fill(0.0)
    api.assemble(b, api.LinearForm(op, api.DataFunction.polynomial(terms, dim, 1)))
    assert np.max(np.abs(b.entries - ref)) <= 1e-12 * np.max(np.abs(ref))
