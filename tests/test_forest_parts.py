"""Batches that a budget splits into parts: bits as in one part, as few parts as
fit, and budgets below the bound of the large fronts' buffers that hold the
whole batch keep it in one.

The number of parts shows in the launches of a solve: every part has launches
of its own, an unsplit batch has those of one."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [9, 30, 3, 30, 16, 28, 30, 30]


def _solve(G, ctx, again=False):
    from grmp_gb300 import stokes as S
    prob = S.make_batch(sizes=np.array(SIZES), nus=np.geomspace(0.1, 1.0, len(SIZES)), seed=11)
    sysd = S.StokesBatchSystem(ctx, prob, mixed=False, direct=True)
    sysd.assemble()
    n0, n1 = ctypes.c_uint64(), ctypes.c_uint64()
    ctx.check(ctx.lib.grmp_context_launches(ctx.h, ctypes.byref(n0)))
    sysd.solve(sweeps=3, reltol=1e-12)
    ctx.check(ctx.lib.grmp_context_launches(ctx.h, ctypes.byref(n1)))
    return sysd, n1.value - n0.value


def test_one_part_where_all_fits(G, ctx):
    sysd, launches = _solve(G, ctx)
    u, p = sysd.velocity().copy(), sysd.pressure().copy()
    c = G.GB300Context(0, hbm_budget_bytes=600 << 20)
    small, n = _solve(G, c)
    assert n == launches
    assert np.array_equal(small.velocity(), u) and np.array_equal(small.pressure(), p)


def test_parts_of_several_problems(G, ctx):
    sysd, one = _solve(G, ctx)
    u, p = sysd.velocity().copy(), sysd.pressure().copy()
    counts = []
    for mb in (300, 200, 140, 110, 90, 75, 60, 50, 40):
        c = G.GB300Context(0, hbm_budget_bytes=mb << 20)
        try:
            small, n = _solve(G, c)
        except G.GrmpError as e:
            assert "BUDGET" in str(e)   # not even one problem at a time
            break
        assert np.array_equal(small.velocity(), u) and np.array_equal(small.pressure(), p)
        counts.append(n)
    # less room, more parts; and between one part and a part for each problem there are others
    assert counts == sorted(counts)
    assert len(set(counts)) >= 3, (one, counts)
