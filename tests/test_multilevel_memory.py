"""The hierarchy under a budget: a shortage that passes is forgotten, and of two
precisions that do not fit together each has the room when it is asked for.

Budgets come from what the same calls take in a context without one.  Solutions
are compared bit for bit with those of that context: with enough room the
solver is the same one, and every sum has a fixed order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 60   # 14,641 P2 rows: no timed choice of a Jacobi configuration


class _Problem:
    def __init__(self, G, ctx):
        from grmp_gb300 import fespace as F
        self.G, self.ctx = G, ctx
        g = G.grid_unitsquare(N)
        self.S = F.FESpace(F.H1P2(1, 2), g)
        kappa = np.exp(np.random.default_rng(3).standard_normal(g.ncells))
        self.ops = [G.BilinearForm([G.Gradient, G.Gradient], G.CellCoefficient(kappa), APT=G.APT_SymmetricBilinearForm)]
        self.A = G.FEMatrix(ctx, self.S, self.ops)
        self.b, self.x = G.FEVector(ctx, self.S), G.FEVector(ctx, self.S)
        G.assemble(self.A, self.ops, G.FP64_FP32)
        self.b.upload(np.random.default_rng(4).standard_normal(self.S.ndofs))
        G.apply_dirichlet(self.A, self.b, self.S.boundary_dofs(), None, G.DIRICHLET_ELIMINATE)

    def solve(self, mode):
        st = self.G.GB300PCG(mode=mode, reltol=1e-11, abstol=0.0).solve(self.A, self.b, self.x)
        assert st["final_relres"] <= 1e-10
        return st["spmv_config"] >= 90000, self.x.entries.copy()


def _sizes(G):
    """Memory before the solves, with the FP64 storage, with both."""
    c = G.GB300Context(0)
    p = _Problem(G, c)
    base = c.memory_in_use()
    took64, x64 = p.solve("fp64")
    one = c.memory_in_use()
    took32, x32 = p.solve("mixed")
    assert took64 and took32
    return base, one, c.memory_in_use(), x64, x32


def _vector(G, ctx, bytes_):
    class S:
        ndofs = int(bytes_) // 8
    return G.FEVector(ctx, S)


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_a_shortage_that_passes(G, mode):
    base, one, both, x64, x32 = _sizes(G)
    c = G.GB300Context(0, hbm_budget_bytes=both + (8 << 20))
    p = _Problem(G, c)
    hold = _vector(G, c, both + (8 << 20) - base - (3 << 20))   # 3 MB left: the Jacobi workspace
    assert not p.solve(mode)[0]
    del hold
    took, x = p.solve(mode)
    assert took and np.array_equal(x, x64 if mode == "fp64" else x32)


def test_two_precisions_in_turn(G):
    base, one, both, x64, x32 = _sizes(G)
    c = G.GB300Context(0, hbm_budget_bytes=one + (both - one) // 2)
    p = _Problem(G, c)
    for mode in ("fp64", "mixed", "fp64", "mixed", "mixed", "fp64"):
        took, x = p.solve(mode)
        assert took and np.array_equal(x, x64 if mode == "fp64" else x32)


def test_storage_that_does_not_fit_leaves_the_other(G):
    """Room for the FP32 hierarchy and the FP64 Jacobi workspace, not for the
    FP64 hierarchy."""
    base, one, both, x64, x32 = _sizes(G)
    c0 = G.GB300Context(0)
    p = _Problem(G, c0)
    p.solve("mixed")
    only32 = c0.memory_in_use()
    G.GB300PCG(mode="fp64", reltol=1e-11, abstol=0.0, spmv_config=404).solve(p.A, p.b, p.x)
    budget = c0.memory_in_use() + (64 << 10)
    assert only32 < budget < one
    c = G.GB300Context(0, hbm_budget_bytes=budget)
    p = _Problem(G, c)
    for mode, fits in (("mixed", True), ("fp64", False), ("mixed", True), ("fp64", False)):
        took, x = p.solve(mode)
        assert took == fits
        assert not fits or np.array_equal(x, x32)


def test_the_jacobi_workspace_comes_first(G):
    """Room for the FP32 hierarchy alone: the FP64 solve takes its memory."""
    base, one, both, x64, x32 = _sizes(G)
    c0 = G.GB300Context(0)
    p = _Problem(G, c0)
    p.solve("mixed")
    c = G.GB300Context(0, hbm_budget_bytes=c0.memory_in_use() + (64 << 10))
    p = _Problem(G, c)
    assert p.solve("mixed")[0]
    assert not p.solve("fp64")[0]
    p.solve("mixed")


def test_memory_goes_to_what_is_allocated_later(G):
    """A vector and a second matrix that fit beside the first matrix, not beside
    its hierarchy too: they are had, and the hierarchy is made again when they are gone."""
    base, one, both, x64, x32 = _sizes(G)
    budget = one + (1 << 20)
    c = G.GB300Context(0, hbm_budget_bytes=budget)
    p = _Problem(G, c)
    assert p.solve("fp64")[0]
    big = _vector(G, c, budget - base - (1 << 20))
    big.fill(2.0)
    took, x = p.solve("fp64")   # the Jacobi workspace fits beside the vector
    assert not took and np.linalg.norm(x - x64) <= 1e-8 * np.linalg.norm(x64)
    assert np.array_equal(big.entries, np.full(big.n, 2.0))
    del big
    took, x = p.solve("fp64")
    assert took and np.array_equal(x, x64)
    for _ in range(3):   # again and again: then the analysis is no longer made for one solve each
        big = _vector(G, c, budget - base - (1 << 20))
        del big
        took, x = p.solve("fp64")
    assert not took and np.linalg.norm(x - x64) <= 1e-8 * np.linalg.norm(x64)
    A2 = G.FEMatrix(c, p.S, p.ops)
    G.assemble(A2, p.ops, G.FP64)
    y = G.FEVector(c, p.S)
    G.spmv(A2, p.x, y, G.FP64)
    assert np.all(np.isfinite(y.entries))

