"""Nested-dissection ordering on patterns of every shape it can meet: no
separator at all (complete graphs, stars), long thin ones (paths, strips),
several components, isolated DoFs, sizes around the leaf size; the direct
solve of an imported matrix on each against numpy's dense solve."""
import numpy as np
import pytest


def _laplacian(n, edges):
    A = np.eye(n) * 0.5
    for i, j in edges:
        A[i, i] += 1
        A[j, j] += 1
        A[i, j] -= 1
        A[j, i] -= 1
    return A


def _grid(nx, ny):
    e = [(y * nx + x, y * nx + x + 1) for y in range(ny) for x in range(nx - 1)]
    return nx * ny, e + [(y * nx + x, y * nx + x + nx) for y in range(ny - 1) for x in range(nx)]


def _pattern(name):
    if name.startswith("path"):
        n = int(name[4:])
        return n, [(i, i + 1) for i in range(n - 1)]
    if name == "star":
        return 120, [(0, i) for i in range(1, 120)]
    if name == "complete":
        return 70, [(i, j) for i in range(70) for j in range(i)]
    if name == "strip":
        return _grid(3, 150)
    if name == "square":
        return _grid(23, 21)
    if name == "two components and isolated":
        n1, e1 = _grid(9, 11)
        n2, e2 = _grid(30, 4)
        return n1 + n2 + 5, e1 + [(i + n1, j + n1) for i, j in e2]
    if name == "isolated":
        return 60, []
    rng = np.random.default_rng(3)
    return 200, [(i, j) for i in range(200) for j in range(i) if rng.random() < 0.02]


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["direct", "mixed_direct"])
@pytest.mark.parametrize("name", ["path1", "path48", "path49", "path300", "star", "complete", "strip", "square",
                                  "two components and isolated", "isolated", "random"])
def test_direct_solve_on_pattern(G, ctx, name, mode):
    """Diagonally dominant matrices, condition at most 2 * 240 + 1 (the star's
    hub), so n cond eps < 1e-10 bounds both solutions."""
    sp = pytest.importorskip("scipy.sparse")
    n, edges = _pattern(name)
    A = _laplacian(n, edges)
    x0 = np.random.default_rng(1).standard_normal(n)
    M = G.ImportedMatrix(ctx, sp.csc_matrix(A))

    class S:
        ndofs = n
    b, x = G.FEVector(ctx, S), G.FEVector(ctx, S)
    b.upload(A @ x0)
    G.GB300PCG(mode=mode, reltol=1e-13, abstol=0.0, maxiter=200).solve(M, b, x)
    assert np.linalg.norm(x.entries - x0) <= 1e-10 * np.linalg.norm(x0)
