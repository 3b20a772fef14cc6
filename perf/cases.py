"""What the speed of this framework is measured on.

Each case is one pass that a user's program makes through the public Python
entry points (the ctypes mirror of the C-ABI): assemble and solve, a batch of
Stokes problems, a Newton step, a reconstructed right-hand side, the assembly
and estimator pass of a stabilised problem, a burst of served requests.
Meshes, spaces, patterns and solver handles are kept by such a program and are
made in prepare(); everything that depends on the data of the pass (coefficients,
forces, iterates) is taken from the seed and goes through run() every time.

exact() restates every discrete problem in 64 bits with plain torch and numpy.
"""
import functools
import importlib.util
import itertools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.getcwd()


def _package():
    """The package directory's name holds a dot: it is imported as grmp_gb300."""
    if "grmp_gb300" not in sys.modules:
        d = os.path.join(ROOT, "gradientrobustmultiphysics.jl_gb300")
        spec = importlib.util.spec_from_file_location("grmp_gb300", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["grmp_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["grmp_gb300"]


_package()


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest assemble-and-solve (1,089 DoFs, the smoke problem): launches, copies and latency
        dict(name="poisson2d-P2-16-mixed", kind="poisson", dim=2, order=2, n=16, mode="mixed", coef="constant"),
        # 2D P2 Poisson 128 x 128 with constant diffusion 1e-3: in L2, many short iterations
        dict(name="poisson2d-P2-128-mixed", kind="poisson", dim=2, order=2, n=128, mode="mixed", coef="constant"),
        # the headline: 3D P2 Poisson on 64^3 Kuhn cubes, per-cell lognormal diffusion, 2.1M DoFs
        dict(name="poisson3d-P2-64-mixed", kind="poisson", dim=3, order=2, n=64, mode="mixed", coef="lognormal"),
        # the plain FP64 path, first order, an odd size
        dict(name="poisson3d-P1-61-fp64", kind="poisson", dim=3, order=1, n=61, mode="fp64", coef="lognormal"),
        # nearly incompressible elasticity 256 x 256 (526k DoFs): FP32 factor, FP64 conjugate gradients
        dict(name="elasticity2d-256-mixed_direct", kind="elasticity", n=256, mode="mixed_direct"),
        # the FP64 direct solver (the reference's default kind of solve), an ordinary odd size
        dict(name="elasticity2d-45-direct", kind="elasticity", n=45, mode="direct"),
        # batched gradient-robust Stokes, 8 x 8 to 96 x 96 squares
        dict(name="stokes2d-160", kind="stokes", dim=2, nprob=160, nmin=8, nmax=96, draw=0),
        # the same in 3D, 2^3 to 6^3 cubes
        dict(name="stokes3d-96", kind="stokes", dim=3, nprob=96, nmin=2, nmax=6, draw=0),
        # one Newton step of nonlinear diffusion (Example205's kernel) with its non-symmetric solve
        dict(name="newton2d-P2-41", kind="newton", dim=2, order=2, n=41, form="diffusion"),
        # reconstructed right-hand side on a 3D Bernardi-Raugel space
        dict(name="recon3d-BDM1-24", kind="recon", dim=3, n=24, target="BDM1"),
        # gradient-jump stabilised operator, its application, error and jump estimators (2D P2)
        dict(name="estimate2d-P2-180", kind="estimate", dim=2, order=2, n=180),
        # a burst of pooled requests at the serving engine: P1 / P2, 2D / 3D, 1e3 to 1e5 DoFs
        dict(name="serve-12", kind="serve", nreq=12, nmeshes=6, dofs_max=100000, draw=3),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "poisson", "elasticity", "stokes", "newton", "recon", "estimate", "serve"])
    if kind == "poisson":
        dim, order = rng.choice([2, 3]), rng.choice([1, 2])
        n = _logint(rng, 8, 250 // order) if dim == 2 else _logint(rng, 4, 92 // order)
        return dict(kind=kind, dim=dim, order=order, n=n, mode=rng.choice(["fp64", "mixed"]),
                    coef=rng.choice(["constant", "lognormal"]))
    if kind == "elasticity":
        mode = rng.choice(["direct", "mixed_direct"])
        return dict(kind=kind, n=_logint(rng, 10, 60 if mode == "direct" else 200), mode=mode)
    if kind == "stokes":
        dim = rng.choice([2, 3])
        nmin = rng.randint(2, 16) if dim == 2 else 2
        # batches of small squares only, or with large ones among them
        nmax = rng.choice([rng.randint(nmin + 8, 28), rng.randint(52, 72)]) if dim == 2 else rng.randint(3, 6)
        return dict(kind=kind, dim=dim, nprob=_logint(rng, 8, 128), nmin=nmin, nmax=nmax, draw=rng.randint(0, 999))
    if kind == "newton":
        form = rng.choice(["diffusion", "grad_diffusion", "convection"])
        order = rng.choice([1, 2])
        return dict(kind=kind, dim=2, order=order, n=_logint(rng, 10, (60 if form == "convection" else 90) // order),
                    form=form)
    if kind == "recon":
        dim = rng.choice([2, 3])
        target = rng.choice(["RT0", "BDM1", "RT1", "BDM2"] if dim == 2 else ["RT0", "BDM1"])
        return dict(kind=kind, dim=dim, n=_logint(rng, 10, 220) if dim == 2 else _logint(rng, 4, 24), target=target)
    if kind == "estimate":
        dim, order = rng.choice([2, 3]), rng.choice([1, 2])
        n = _logint(rng, 10, 220) if dim == 2 else _logint(rng, 4, 40 // (2 * order))
        return dict(kind=kind, dim=dim, order=order, n=n)
    return dict(kind=kind, nreq=rng.randint(4, 12), nmeshes=rng.randint(2, 6), dofs_max=_logint(rng, 10000, 100000),
                draw=rng.randint(0, 999))


# ------------------------------------------------------------------ meshes (the user's own arrays)
@functools.lru_cache(maxsize=256)
def _grid(dim, n):
    G = _package()
    return G.grid_unitsquare(n) if dim == 2 else G.grid_unitcube_kuhn(n)


@functools.lru_cache(maxsize=16)
def _space(kind, dim, n):
    """Host-built spaces (the elements whose DoF maps need faces)."""
    G = _package()
    return G.FESpace(G.H1BR(dim) if kind == "BR" else G.H1P2B(2, 2), _grid(dim, n))


@functools.lru_cache(maxsize=16)
def _batch(dim, nprob, nmin, nmax, draw_):
    from grmp_gb300 import stokes as S
    rng = np.random.default_rng(draw_)
    sizes = np.rint(np.exp(rng.uniform(np.log(nmin), np.log(nmax), nprob))).astype(int)
    sizes[0] = nmax
    bm = S.BatchedMesh([_grid(dim, int(n)) for n in sizes])
    return sizes, bm, S.BatchedBRSpace(bm)


class _DeviceArray:
    """A library vector as a torch tensor without a copy; keeps the vector."""

    def __init__(self, v):
        import ctypes
        self.keep = v
        p = ctypes.c_void_p()
        v.ctx.check(v.ctx.lib.grmp_vector_device_ptr(v.h, ctypes.byref(p)))
        self.__cuda_array_interface__ = {"shape": (int(v.n),), "typestr": "<f8", "data": (p.value, False),
                                         "version": 3, "strides": None}


def _tensor(v):
    return torch.as_tensor(_DeviceArray(v), device="cuda:0")


def _fixed_elasticity(n, ndofs):
    """DoFs of both components on the left edge x = 0 (vertices, then edges)."""
    coords, cells = _grid(2, n).coords, _grid(2, n).cells
    cd, edges, nd = _dofmap(2, 2, 1, n)
    x = np.concatenate([coords[:, 0], coords[edges].mean(axis=1)[:, 0]])
    f = np.flatnonzero(np.abs(x) < 1e-12)
    return np.concatenate([f, f + nd]).astype(np.int32)


# ------------------------------------------------------------------ data of a pass
def _fourier(rng, dim):
    return rng.standard_normal(8), rng.integers(1, 5, size=(8, dim)).astype(np.float64)


def _data(case, seed):
    rng = np.random.default_rng([seed, 77])
    k = case["kind"]
    if k == "poisson":
        ncells = (2 if case["dim"] == 2 else 6) * case["n"] ** case["dim"]
        amp, modes = _fourier(rng, case["dim"])
        kappa = np.exp(rng.standard_normal(ncells)) if case["coef"] == "lognormal" else np.full(ncells, 1e-3)
        return dict(kappa=kappa, amp=amp, k=modes)
    if k == "elasticity":
        return dict(force=rng.standard_normal((2 * case["n"] ** 2, 2)))
    if k == "stokes":
        from grmp_gb300 import stokes as S
        sizes = _batch(case["dim"], case["nprob"], case["nmin"], case["nmax"], case["draw"])[0]
        nus = np.exp(rng.uniform(np.log(1e-2), 0.0, len(sizes)))
        if case["dim"] == 2:
            terms = np.stack([S.grad_plus_curl_terms(S.cubic_coefficients(rng), S.cubic_coefficients(rng)) for _ in sizes])
        else:
            terms = np.stack([S.grad_plus_curl_terms_3d(S.cubic_coefficients_3d(rng),
                                                        [S.cubic_coefficients_3d(rng) for _ in range(3)]) for _ in sizes])
        return dict(nus=nus, terms=terms)
    if k == "newton":
        # a smooth iterate with a small rough part, as in the middle of a Newton loop
        nc = 2 if case["form"] == "convection" else 1
        amp, modes = _fourier(rng, 2)
        X = _dof_points(2, case["order"], case["n"])
        u = np.concatenate([sum(0.3 * a * np.sin(np.pi * (X @ m) + c) for a, m in zip(amp, modes)) for c in range(nc)])
        return dict(u=u + 0.01 * rng.standard_normal(u.size), f=np.concatenate([10.0 + rng.standard_normal(1), -rng.random(1)])[:nc])
    if k == "recon":
        e = [p for p in itertools.product(range(3), repeat=case["dim"]) if sum(p) <= 2]
        return dict(terms=np.array([(c, rng.standard_normal(), *p, *([0] * (3 - case["dim"])))
                                    for c in range(case["dim"]) for p in e]))
    if k == "estimate":
        nd = _dofmap(case["dim"], case["order"], 1, case["n"])[2]
        d = case["dim"]
        lin = np.array([(c, rng.standard_normal(), *[int(i == j) for i in range(3)]) for c in range(d) for j in range(d)])
        return dict(u=rng.standard_normal(nd), kappa=np.exp(rng.standard_normal(_grid(d, case["n"]).ncells)), terms=lin)
    if k == "serve":
        pool = np.random.default_rng(case["draw"])
        meshes = []
        for _ in range(case["nmeshes"]):
            dim, order = int(pool.integers(2, 4)), int(pool.integers(1, 3))
            dofs = math.exp(pool.uniform(math.log(1e3), math.log(case["dofs_max"])))
            meshes.append((dim, order, max(2, int(round((dofs ** (1.0 / dim) - 1) / order))), bool(pool.random() < 0.5)))
        reqs = []
        for i in range(case["nreq"]):
            dim, order, n, reaction = meshes[int(pool.integers(0, len(meshes)))]
            amp, modes = _fourier(rng, dim)
            reqs.append(dict(dim=dim, order=order, n=n, alpha=float(rng.uniform(0.1, 10)) if reaction else 0.0,
                             kappa=np.exp(rng.standard_normal(_grid(dim, n).ncells)), amp=amp, k=modes))
        return dict(reqs=reqs)
    raise ValueError(k)


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    G = _package()
    D = _data(case, seed)
    k = case["kind"]
    if k == "serve":
        from grmp_gb300 import serve as S
        reqs = []
        for r in D["reqs"]:
            g = _grid(r["dim"], r["n"])
            FES = _serve_space(r["dim"], r["order"], r["n"])
            reqs.append(S.ServeRequest(r["dim"], r["order"], r["n"], FES, r["kappa"], r["alpha"], r["amp"], r["k"],
                                       FES.boundary_dofs(), mesh_key=S.mesh_key(r["dim"], r["n"], r["order"])))
        return dict(case=case, srv=S.Server(0, 150 << 30, 4), reqs=reqs)
    ctx = G.GB300Context(0)
    s = dict(case=case, ctx=ctx)
    if k in ("poisson", "elasticity"):
        dim = case.get("dim", 2)
        g = _grid(dim, case["n"])
        if k == "poisson":
            fe = G.H1P1(1) if case["order"] == 1 else G.H1P2(1, dim)
            if case["coef"] == "constant":
                ops = [G.LaplaceOperator(1e-3)]
            else:
                ops = [G.BilinearForm([G.Gradient, G.Gradient], G.CellCoefficient(D["kappa"]),
                                      APT=G.APT_SymmetricBilinearForm)]
            rhs = G.LinearForm(G.Identity, G.DataFunction.fourier(D["amp"], D["k"]))
            reltol = 1e-11
        else:
            fe, ops = G.H1P2(2, 2), [G.HookStiffnessOperator2D(1.0, 1e3)]
            rhs = G.LinearForm(G.Identity, G.DataFunction.cellwise(D["force"]))
            reltol = 1e-12
        FES = ctx.space_on_device(fe, g, download=False)
        s["fixed"] = ctx.boundary_dofs(FES) if k == "poisson" else _fixed_elasticity(case["n"], FES.ndofs)
        s["ops"], s["rhs"] = ops, rhs
        s["prec"] = G.FP64_FP32 if case["mode"] == "mixed" else G.FP64
        s["solver"] = G.GB300PCG(mode=case["mode"], reltol=reltol, abstol=0.0)
        s["A"] = G.FEMatrix(ctx, FES, ops)
        s["b"], s["x"] = G.FEVector(ctx, FES), G.FEVector(ctx, FES)
        s["out"] = _tensor(s["x"])
    elif k == "stokes":
        from grmp_gb300 import stokes as S
        sizes, bm, V = _batch(case["dim"], case["nprob"], case["nmin"], case["nmax"], case["draw"])
        s["sys"] = S.StokesBatchSystem(ctx, S.StokesBatchProblem(sizes, D["nus"], D["terms"], bm, V, 1e4),
                                       mixed=False, direct=True)
        s["out"] = (_tensor(s["sys"].u), _tensor(s["sys"].p))
    elif k == "newton":
        nc = 2 if case["form"] == "convection" else 1
        FES = ctx.space_on_device(G.H1P1(nc) if case["order"] == 1 else G.H1P2(nc, 2), _grid(2, case["n"]), download=False)
        s["fixed"] = ctx.boundary_dofs(FES)
        s["ops"] = [G.LaplaceOperator(1.0), G.StructuralCoupling()]
        s["form"] = G.NonlinearForm(case["form"], kappa=1.0, beta=1.0, bonus_quadorder=2)
        s["rhs"] = G.LinearForm(G.Identity, G.DataFunction.constant(D["f"]))
        s["solver"] = G.GB300PCG(mode="bicgstab", reltol=1e-11, abstol=0.0)
        s["A"] = G.FEMatrix(ctx, FES, s["ops"])
        s["b"], s["u"], s["x"] = (G.FEVector(ctx, FES) for _ in range(3))
        s["u"].upload(D["u"])
        s["out"] = _tensor(s["x"])
    elif k == "recon":
        p2b = case["target"] in ("RT1", "BDM2")
        FES = _space("P2B" if p2b else "BR", case["dim"], case["n"])
        from grmp_gb300 import api
        op = {"RT0": api.ReconstructionIdentity, "BDM1": api.ReconstructionIdentityBDM1,
              "RT1": api.ReconstructionIdentityRT1, "BDM2": api.ReconstructionIdentityBDM2}[case["target"]]
        s["lf"] = G.LinearForm(op, G.DataFunction.polynomial(D["terms"], case["dim"], bonus_quadorder=2 if p2b else 1))
        s["b"] = G.FEVector(ctx, FES)
        ctx.space(FES)
        s["out"] = _tensor(s["b"])
    elif k == "estimate":
        dim, order = case["dim"], case["order"]
        g = _grid(dim, case["n"])
        FES = ctx.space_on_device(G.H1P1(1) if order == 1 else G.H1P2(1, dim), g, download=False)
        lap = G.BilinearForm([G.Gradient, G.Gradient], G.CellCoefficient(D["kappa"]), APT=G.APT_SymmetricBilinearForm)
        jump = G.BilinearForm([G.Jump(G.Gradient), G.Jump(G.Gradient)], G.FaceVolumePower(2.0), AT=G.ON_IFACES, factor=0.1)
        s["ops"] = [lap, jump]
        s["A"] = G.FEMatrix(ctx, FES, s["ops"])
        s["u"], s["y"] = G.FEVector(ctx, FES), G.FEVector(ctx, FES)
        s["u"].upload(D["u"])
        s["err"] = G.L2ErrorIntegrator(G.DataFunction.polynomial(D["terms"], dim, bonus_quadorder=1), G.Gradient)
        s["jumps"] = G.FaceJumpIntegrator(normal=True, power=1.0)
        s["out"] = _tensor(s["y"])
    return s


@functools.lru_cache(maxsize=64)
def _serve_space(dim, order, n):
    G = _package()
    return G.FESpace(G.H1P1(1) if order == 1 else G.H1P2(1, dim), _grid(dim, n))


# ------------------------------------------------------------------ run
def run(s):
    G = _package()
    k = s["case"]["kind"]
    if k in ("poisson", "elasticity"):
        # solve!: assembly, right-hand side, boundary data, solver
        G.assemble(s["A"], s["ops"], s["prec"])
        s["b"].fill(0.0)
        G.assemble(s["b"], s["rhs"])
        G.apply_dirichlet(s["A"], s["b"], s["fixed"])
        s["solver"].solve(s["A"], s["b"], s["x"])
        return s["out"]
    if k == "stokes":
        s["sys"].assemble()
        s["sys"].solve(sweeps=6, reltol=1e-12, maxiter=1, sweep_tol=0.0)
        return s["out"]
    if k == "newton":
        # one step of solve_nonlinear
        G.assemble(s["A"], s["ops"], G.FP64)
        s["b"].fill(0.0)
        G.assemble(s["b"], s["rhs"])
        G.assemble_nonlinear(s["A"], s["b"], s["u"], s["form"], G.FP64, add=True)
        G.apply_dirichlet(s["A"], s["b"], s["fixed"])
        s["solver"].solve(s["A"], s["b"], s["x"])
        return s["out"]
    if k == "recon":
        s["b"].fill(0.0)
        G.assemble(s["b"], s["lf"])
        return s["out"]
    if k == "estimate":
        G.assemble(s["A"], s["ops"], G.FP64)
        G.spmv(s["A"], s["u"], s["y"], G.FP64)
        return s["out"], s["err"].evaluate_cells(s["u"]), s["jumps"].evaluate_faces(s["u"])
    # serve: the burst is submitted and every answer waited for
    ids = [s["srv"].submit(r, "mixed", 1e-11) for r in s["reqs"]]
    out = []
    for r, i in zip(s["reqs"], ids):
        rc, x, st = s["srv"].wait(i, r.ndofs)
        if rc:
            raise RuntimeError("a served request failed with %d" % rc)
        out.append(x)
    return out


# ------------------------------------------------------------------ work
def _sizes(dim, order, nc, n):
    """(cells, DoFs, nonzeros of a structured mesh's matrix, about)"""
    cells = (2 if dim == 2 else 6) * n ** dim
    dofs = nc * (order * n + 1) ** dim
    per = {(2, 1): 5, (2, 2): 10, (3, 1): 7.5, (3, 2): 26}[(dim, order)]
    return cells, dofs, int(per * nc * dofs)


def work(case):
    """Bytes: the data of the pass, the mesh and DoF map read once, the matrix
    values and the result written once.  Flops: the element contractions and
    the solver's multiply-adds at the iteration counts (or front sizes) that
    the method needs on these meshes."""
    k = case["kind"]
    if k in ("poisson", "elasticity", "newton", "estimate"):
        dim, order, n = case.get("dim", 2), case.get("order", 2), case["n"]
        nc = 2 if k == "elasticity" or case.get("form") == "convection" else 1
        cells, dofs, nnz = _sizes(dim, order, nc, n)
        ld = nc * {(2, 1): 3, (2, 2): 6, (3, 1): 4, (3, 2): 10}[(dim, order)]
        b = cells * (8 + 4 * (dim + 1) + 4 * ld) + 8 * dim * (n + 1) ** dim + 8 * nnz + 8 * dofs
        f = cells * ld * ld * dim * (dim + 1)
        if k == "poisson":
            its = (8 if dim == 2 else 15) * n * order // 2
            f += its * (2 * nnz + 10 * dofs)
        elif k == "newton":
            f += cells * ld * ld * 50 + 4 * n * (4 * nnz + 20 * dofs)
        elif k == "elasticity":
            f += 10.0 * dofs ** 1.5 * 8
        else:
            b += 8 * (dofs + 3 * cells)
            f += cells * (dim + 1) * 4 * ld * ld
        return {"bytes": float(b), "flops": float(f)}
    if k == "stokes":
        b = f = 0.0
        for n in _batch(case["dim"], case["nprob"], case["nmin"], case["nmax"], case["draw"])[0]:
            n = int(n)
            dofs = 2 * (n + 1) ** 2 + 3 * n * n + 2 * n if case["dim"] == 2 else 3 * (n + 1) ** 3 + 12 * n ** 3 + 6 * n * n
            cells = 2 * n * n if case["dim"] == 2 else 6 * n ** 3
            b += cells * 150.0 + dofs * (8 * 15 + 16)
            f += 30.0 * dofs ** 1.5 if case["dim"] == 2 else 5.0 * dofs ** 2
        return {"bytes": b, "flops": f}
    if k == "recon":
        cells = (2 if case["dim"] == 2 else 6) * case["n"] ** case["dim"]
        ld = 14 if case["target"] in ("RT1", "BDM2") else (9 if case["dim"] == 2 else 16)
        return {"bytes": cells * (4.0 * ld + 12 * (case["dim"] + 1) + 8 * case["dim"]) + 8.0 * cells * ld / 4,
                "flops": cells * ld * (400.0 if case["dim"] == 2 else 600.0)}
    b = f = 0.0
    for r in _data(case, 0)["reqs"]:
        w = work(dict(kind="poisson", dim=r["dim"], order=r["order"], n=r["n"]))
        b, f = b + w["bytes"], f + w["flops"]
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact: 64 bits, plain torch and numpy
_EDGES = {2: [(0, 1), (1, 2), (2, 0)], 3: [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]}
_FACES = {2: [(0, 1), (1, 2), (2, 0)], 3: [(0, 1, 2), (0, 1, 3), (1, 2, 3), (0, 2, 3)]}


def _entities(cells, local):
    """Distinct sorted vertex tuples in lexicographic order, and each cell's numbers of them."""
    t = np.sort(cells[:, np.array(local)], axis=2).astype(np.int64)
    base = int(cells.max()) + 1
    key = np.zeros(t.shape[:2], dtype=np.int64)
    for j in range(t.shape[2]):
        key = key * base + t[:, :, j]
    _, first, inv = np.unique(key.ravel(), return_index=True, return_inverse=True)
    return t.reshape(-1, t.shape[2])[first], inv.reshape(key.shape)


@functools.lru_cache(maxsize=8)
def _dofmap(dim, order, nc, n):
    """(cell DoFs, edge vertices, DoFs of one component): vertices, then edges, component by component."""
    g = _grid(dim, n)
    cells = g.cells.astype(np.int64)
    nv = g.coords.shape[0]
    cd, edges, nd = cells, np.zeros((0, 2), dtype=np.int64), nv
    if order == 2:
        edges, ce = _entities(cells, _EDGES[dim])
        cd, nd = np.concatenate([cells, ce + nv], axis=1), nv + edges.shape[0]
    return np.concatenate([cd + c * nd for c in range(nc)], axis=1), edges, nd


def _dof_points(dim, order, n):
    X = _grid(dim, n).coords
    e = _dofmap(dim, order, 1, n)[1]
    return np.concatenate([X, X[e].mean(axis=1)]) if order == 2 else X


def _boundary(X):
    """Points on the boundary of the unit square or cube."""
    return np.flatnonzero((np.minimum(X, 1 - X) < 1e-12).any(axis=1))


def _duffy(dim, degree):
    """A rule on the reference simplex, exact to the degree; weights sum to 1."""
    x, w = np.polynomial.legendre.leggauss(degree // 2 + 2)
    x, w = (x + 1) / 2, w / 2
    P, W = [], []
    for idx in itertools.product(range(len(x)), repeat=dim):
        a = [x[i] for i in idx]
        wt = np.prod([w[i] for i in idx])
        if dim == 1:
            P.append((a[0],))
        elif dim == 2:
            P.append((a[0], a[1] * (1 - a[0])))
            wt *= 2 * (1 - a[0])
        else:
            P.append((a[0], a[1] * (1 - a[0]), a[2] * (1 - a[0]) * (1 - a[1])))
            wt *= 6 * (1 - a[0]) ** 2 * (1 - a[1])
        W.append(wt)
    return np.array(P), np.array(W)


def _rhs_rule(dim, order):
    """The rules that linear forms use at the element's own order (1 or 2)."""
    if order == 1:
        return np.full((1, dim), 1.0 / (dim + 1)), np.ones(1)
    if dim == 2:
        return np.array([[0.5, 0.5], [0.0, 0.5], [0.5, 0.0]]), np.full(3, 1 / 3)
    a, b = 0.1381966011250105, 0.5854101966249685
    return np.array([[a, a, a], [b, a, a], [a, b, a], [a, a, b]]), np.full(4, 0.25)


def _basis(dim, order, x):
    """Values [q, a] and reference derivatives [q, a, dim] of P1 / P2."""
    lam = np.concatenate([1 - x.sum(axis=1, keepdims=True), x], axis=1)
    dl = np.concatenate([-np.ones((1, dim)), np.eye(dim)])
    if order == 1:
        return lam, np.broadcast_to(dl, (x.shape[0], dim + 1, dim)).copy()
    v = [lam[:, i] * (2 * lam[:, i] - 1) for i in range(dim + 1)]
    d = [(4 * lam[:, i] - 1)[:, None] * dl[i] for i in range(dim + 1)]
    for a, b in _EDGES[dim]:
        v.append(4 * lam[:, a] * lam[:, b])
        d.append(4 * (lam[:, a, None] * dl[b] + lam[:, b, None] * dl[a]))
    return np.stack(v, axis=1), np.stack(d, axis=1)


def _dev():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev())


def _geometry(X, cells):
    P = X[cells]
    A = (P[:, 1:] - P[:, :1]).transpose(1, 2)           # columns x_j - x_0
    det = torch.linalg.det(A)
    return P[:, 0], A, torch.linalg.inv(A).transpose(1, 2), det.abs() / math.factorial(X.shape[1])


def _csr(cd, loc, n):
    """Sum of the local matrices loc[cell, i, j] as a coalesced sparse matrix."""
    ld = cd.shape[1]
    i = cd[:, :, None].expand(-1, -1, ld).reshape(-1)
    j = cd[:, None, :].expand(-1, ld, -1).reshape(-1)
    return torch.sparse_coo_tensor(torch.stack([i, j]), loc.reshape(-1), (n, n)).coalesce()


def _eliminate(M, b, fixed):
    i, v = M.indices(), M.values().clone()
    f = torch.zeros(M.shape[0], dtype=torch.bool, device=v.device)
    f[fixed] = True
    dead = f[i[0]] | f[i[1]]
    v[dead] = 0
    v[dead & (i[0] == i[1])] = 1
    b = b.clone()
    b[fixed] = 0
    return torch.sparse_coo_tensor(i, v, M.shape, is_coalesced=True), b


def _cg(M, b):
    """Jacobi-CG, restarted from the true residual until that no longer falls."""
    A = M.to_sparse_csr()
    i = M.indices()
    d = torch.zeros_like(b).index_add_(0, i[0], torch.where(i[0] == i[1], M.values(), torch.zeros_like(M.values())))
    x, best = torch.zeros_like(b), math.inf
    for _ in range(6):
        r = b - A @ x
        r0 = float(r.norm())
        if r0 >= 0.5 * best or r0 == 0:
            break
        best = r0
        z = r / d
        p, rz = z.clone(), r @ z
        y = torch.zeros_like(b)
        for it in range(20000):
            q = A @ p
            al = rz / (p @ q)
            y += al * p
            r -= al * q
            if it % 25 == 0 and float(r.norm()) <= 1e-9 * r0:
                break
            z = r / d
            rz, old = r @ z, rz
            p = z + (rz / old) * p
        x = x + y
    return x


def _tridiagonal(M, b, line, spd=True):
    """Block tridiagonal solves of M x = b (each DoF couples to the lines next
    to its own): a function that solves for one right-hand side."""
    nl = int(line.max()) + 1
    order = torch.argsort(line, stable=True)
    start = torch.zeros(nl + 1, dtype=torch.int64, device=line.device)
    start[1:] = torch.cumsum(torch.bincount(line, minlength=nl), 0)
    pos = torch.empty_like(order)
    pos[order] = torch.arange(order.numel(), device=line.device)
    i, v = M.indices(), M.values()
    li, lj = line[i[0]], line[i[1]]
    ri, rj = pos[i[0]] - start[li], pos[i[1]] - start[lj]
    st = start.tolist()
    sel = torch.argsort(li * 3 + (lj - li + 1), stable=True)
    cnt = torch.zeros(3 * nl + 1, dtype=torch.int64, device=line.device)
    cnt[1:] = torch.cumsum(torch.bincount(li * 3 + (lj - li + 1), minlength=3 * nl), 0)
    cnt = cnt.tolist()

    def block(k, o):
        e = sel[cnt[3 * k + o + 1]:cnt[3 * k + o + 2]]
        B = torch.zeros(st[k + 1] - st[k], st[k + o + 1] - st[k + o], dtype=v.dtype, device=v.device)
        B[ri[e], rj[e]] = v[e]
        return B

    fac = []          # (factor of the pivot block, lower block, S^-1 upper block)
    for k in range(nl):
        S = block(k, 0)
        if k:
            low = block(k, -1)
            S = S - low @ fac[-1][2]
        else:
            low = None
        F = torch.linalg.cholesky(S) if spd else torch.linalg.lu_factor(S)
        sol = (lambda B, F=F: torch.cholesky_solve(B, F)) if spd else (lambda B, F=F: torch.linalg.lu_solve(*F, B))
        fac.append((sol, low, sol(block(k, 1)) if k + 1 < nl else None))

    def solve(c):
        c = c[order]
        y = []
        for k in range(nl):
            t = c[st[k]:st[k + 1], None]
            if k:
                t = t - fac[k][1] @ y[-1]
            y.append(fac[k][0](t))
        for k in range(nl - 2, -1, -1):
            y[k] = y[k] - fac[k][2] @ y[k + 1]
        x = torch.empty_like(c)
        x[order] = torch.cat(y)[:, 0]
        return x

    A = M.to_sparse_csr()

    def refined(c):
        x = solve(c)
        return x + solve(c - A @ x)
    return refined


def _fourier_at(x, amp, k):
    f = 0
    for a, m in zip(amp, k):
        f = f + float(a) * torch.sin(math.pi * (x @ _t(m)))
    return f


def _exact_poisson(dim, order, n, kappa, alpha, amp, k):
    g = _grid(dim, n)
    cd, _, nd = _dofmap(dim, order, 1, n)
    X, cells, cdt = _t(g.coords), _t(g.cells.astype(np.int64)), _t(cd)
    x0, A, Gm, vol = _geometry(X, cells)
    xq, w = _duffy(dim, 2)
    _, dv = _basis(dim, order, xq)
    K = _t(np.einsum("q,qap,qbs->psab", w, dv, dv))
    C = torch.einsum("ckp,cks,c->cps", Gm, Gm, vol * _t(kappa))
    loc = torch.einsum("cps,psab->cab", C, K)
    if alpha:
        xq, w = _duffy(dim, 4)
        v, _ = _basis(dim, order, xq)
        loc = loc + (alpha * vol)[:, None, None] * _t(np.einsum("q,qa,qb->ab", w, v, v))
    M = _csr(cdt, loc, nd)
    del loc
    xr, w = _rhs_rule(dim, order)
    v, _ = _basis(dim, order, xr)
    b = torch.zeros(nd, dtype=torch.float64, device=X.device)
    for q in range(len(w)):
        f = _fourier_at(x0 + A @ _t(xr[q]), amp, k) * vol * float(w[q])
        b.index_add_(0, cdt.reshape(-1), (f[:, None] * _t(v[q])).reshape(-1))
    M, b = _eliminate(M, b, _t(_boundary(_dof_points(dim, order, n))))
    if dim == 2:
        return _tridiagonal(M, b, _lines(_dof_points(dim, order, n), n))(b)
    return _cg(M, b)


def _lines(X, n):
    return _t(np.floor(X[:, 1] * n + 1e-6).astype(np.int64))


def _exact_elasticity(n, force):
    g = _grid(2, n)
    cd, _, nd = _dofmap(2, 2, 2, n)
    X, cells, cdt = _t(g.coords), _t(g.cells.astype(np.int64)), _t(cd)
    x0, A, Gm, vol = _geometry(X, cells)
    xq, w = _duffy(2, 2)
    _, dv = _basis(2, 2, xq)
    K = torch.einsum("ckp,cls,psab,c->cklab", Gm, Gm, _t(np.einsum("q,qap,qbs->psab", w, dv, dv)), vol)
    mu, lam = 1.0, 1e3
    L = torch.zeros(cells.shape[0], 12, 12, dtype=torch.float64, device=X.device)
    tr = K[:, 0, 0] + K[:, 1, 1]
    for c in range(2):
        for d in range(2):
            B = lam * K[:, c, d] + mu * K[:, d, c]
            if c == d:
                B = B + mu * tr
            L[:, 6 * c:6 * c + 6, 6 * d:6 * d + 6] = B
    M = _csr(cdt, L, 2 * nd)
    xr, w = _rhs_rule(2, 2)
    v, _ = _basis(2, 2, xr)
    m = _t(w @ v)
    b = torch.zeros(2 * nd, dtype=torch.float64, device=X.device)
    lb = (_t(force) * vol[:, None])[:, :, None] * m
    b.index_add_(0, cdt.reshape(-1), lb.reshape(-1))
    M, b = _eliminate(M, b, _t(_fixed_elasticity(n, 2 * nd)))
    line = _lines(_dof_points(2, 2, n), n)
    return _tridiagonal(M, b, torch.cat([line, line]))(b)


def _poly(terms, x, dim):
    f = [0.0 * x[..., 0] for _ in range(dim)]
    for t in terms:
        v = float(t[1])
        for j in range(dim):
            if t[2 + j]:
                v = v * x[..., j] ** int(t[2 + j])
        f[int(t[0])] = f[int(t[0])] + v
    return torch.stack(f, dim=-1)


def _br(dim, g):
    """Bernardi-Raugel data of a mesh: cell DoFs, geometry, the vector basis'
    face normals per cell and the outward fluxes D[c, i, f] of each basis
    function through each local face."""
    coords, cells = g.coords, g.cells.astype(np.int64)
    fv, cf = _entities(cells, _FACES[dim])
    nv, nf = coords.shape[0], fv.shape[0]
    ctr = coords[cells].mean(axis=1)
    nl = dim + 1
    out = np.empty((cells.shape[0], nl, dim))
    area = np.empty((cells.shape[0], nl))
    for f, loc in enumerate(_FACES[dim]):
        P = coords[cells[:, loc]]
        if dim == 2:
            t = P[:, 1] - P[:, 0]
            nn = np.stack([t[:, 1], -t[:, 0]], axis=1)
        else:
            nn = np.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]) / 2
        ar = np.linalg.norm(nn, axis=1)
        nn = nn / ar[:, None]
        sg = np.sign(np.einsum("ij,ij->i", nn, P.mean(axis=1) - ctr))
        out[:, f], area[:, f] = nn * sg[:, None], ar
    # global normal of a face: outward from its first cell
    first = np.full(nf, -1)
    flat = cf.ravel()
    first[flat[::-1]] = np.arange(flat.size)[::-1]
    gn = out.reshape(-1, dim)[first]
    nrm = gn[cf]                                             # [cell, face, dim]
    sign = np.where(np.einsum("cfk,cfk->cf", nrm, out) > 0, 1.0, -1.0)
    cd = np.concatenate([cells + c * nv for c in range(dim)] + [cf + dim * nv], axis=1)
    flux = np.zeros((cells.shape[0], dim * nl + nl, nl))
    for f, loc in enumerate(_FACES[dim]):
        for c in range(dim):
            for a in loc:
                flux[:, c * nl + a, f] = area[:, f] * out[:, f, c] / dim
        flux[:, dim * nl + f, f] = area[:, f] * sign[:, f]
    return cd, cf, nrm, flux, dim * nv + nf


def _br_scalar(dim, x):
    """P1 functions and face bubbles: values and reference derivatives."""
    lam, dl = _basis(dim, 1, x)
    v, d = [lam[:, i] for i in range(dim + 1)], [dl[:, i] for i in range(dim + 1)]
    for loc in _FACES[dim]:
        c = 6.0 if dim == 2 else 60.0
        v.append(c * np.prod(lam[:, loc], axis=1))
        s = 0
        for i in loc:
            s = s + np.prod(lam[:, [j for j in loc if j != i]], axis=1)[:, None] * dl[:, i]
        d.append(c * s)
    return np.stack(v, axis=1), np.stack(d, axis=1)


def _br_rhs(dim, g, terms, target):
    """(f, R v) for one mesh; R v is the RT0 (or BDM1) interpolant of v."""
    cd, cf, nrm, flux, nd = _br(dim, g)
    X, cells, cdt = _t(g.coords), _t(g.cells.astype(np.int64)), _t(cd)
    x0, A, Gm, vol = _geometry(X, cells)
    nl = dim + 1
    opp = [[i for i in range(nl) if i not in loc][0] for loc in _FACES[dim]]
    Xo = X[cells][:, opp]                                    # vertex opposite each face
    fl = _t(flux)
    xq, w = _duffy(dim, 4)
    lb = torch.zeros(cells.shape[0], cd.shape[1], dtype=torch.float64, device=X.device)
    for q in range(len(w)):
        x = x0 + A @ _t(xq[q])
        f = _poly(terms, x, dim) * (vol * float(w[q]))[:, None]
        rt = torch.einsum("cfk,ck->cf", x[:, None] - Xo, f) / (dim * vol)[:, None]   # f . psi_F
        v = torch.einsum("cif,cf->ci", fl, rt)
        if target == "BDM1":                                 # linear fields are their own interpolant
            lam = _basis(dim, 1, xq[q:q + 1])[0][0]
            for c in range(dim):
                v[:, c * nl:(c + 1) * nl] = f[:, c, None] * _t(lam)
        lb += v
    b = torch.zeros(nd, dtype=torch.float64, device=X.device)
    return b.index_add_(0, cdt.reshape(-1), lb.reshape(-1))


def _exact_stokes(case, D):
    dim, lam_ = case["dim"], 1e4
    sizes = _batch(case["dim"], case["nprob"], case["nmin"], case["nmax"], case["draw"])[0]
    U, P = [], []
    cache = {}
    for n, nu, terms in zip(sizes, D["nus"], D["terms"]):
        n = int(n)
        g = _grid(dim, n)
        if n not in cache:
            cd, cf, nrm, flux, nd = _br(dim, g)
            X, cells = _t(g.coords), _t(g.cells.astype(np.int64))
            x0, A, Gm, vol = _geometry(X, cells)
            xq, w = _duffy(dim, 2 if dim == 2 else 4)
            _, dv = _br_scalar(dim, xq)
            K = torch.einsum("ckp,cks,c,psab->cab", Gm, Gm, vol, _t(np.einsum("q,qap,qbs->psab", w, dv, dv)))
            nl = dim + 1
            coef = torch.zeros(cells.shape[0], dim * nl + nl, dim, dtype=torch.float64, device=X.device)
            for c in range(dim):
                coef[:, c * nl:(c + 1) * nl, c] = 1
            coef[:, dim * nl:] = _t(nrm)
            sc = [i % nl for i in range(dim * nl)] + [nl + f for f in range(nl)]
            visc = K[:, sc][:, :, sc] * torch.einsum("cik,cjk->cij", coef, coef)
            div = _t(flux).sum(dim=2)                        # int_T div phi_i
            pts = np.concatenate([g.coords] * dim + [g.coords[_entities(g.cells.astype(np.int64), _FACES[dim])[0]].mean(axis=1)])
            cache[n] = (_t(cd), nd, vol, visc, div, torch.einsum("ci,cj,c->cij", div, div, 1 / vol), pts, _t(_boundary(pts)))
        cd, nd, vol, visc, div, pen, pts, fixed = cache[n]
        f = _br_rhs(dim, g, terms, "RT0")
        M, f0 = _eliminate(_csr(cd, float(nu) * visc + lam_ * pen, nd), f, fixed)
        if dim == 2:
            solve = _tridiagonal(M, f, _lines(pts, n))
        else:
            Lc = torch.linalg.cholesky(M.to_dense())
            Ac = M.to_sparse_csr()

            def solve(b, Lc=Lc, Ac=Ac):
                x = torch.cholesky_solve(b[:, None], Lc)[:, 0]
                return x + torch.cholesky_solve((b - Ac @ x)[:, None], Lc)[:, 0]
        p = torch.zeros(cd.shape[0], dtype=torch.float64, device=f.device)
        for _ in range(6):
            b = f.clone().index_add_(0, cd.reshape(-1), (p[:, None] * div).reshape(-1))
            b[fixed] = 0
            u = solve(b)
            p = p - lam_ * (u[cd] * div).sum(dim=1) / vol
            p = p - (p * vol).sum() / vol.sum()
        U.append(u)
        P.append(p)
    return torch.cat(U), torch.cat(P)


def _exact_newton(case, D):
    order, n, form = case["order"], case["n"], case["form"]
    nc = 2 if form == "convection" else 1
    g = _grid(2, n)
    cd, _, nd = _dofmap(2, order, nc, n)
    X, cells, cdt = _t(g.coords), _t(g.cells.astype(np.int64)), _t(cd)
    x0, A, Gm, vol = _geometry(X, cells)
    nb, ld = cd.shape[1] // nc, cd.shape[1]
    uc = _t(D["u"])[cdt].reshape(-1, nc, nb)
    L = torch.zeros(cells.shape[0], ld, ld, dtype=torch.float64, device=X.device)
    lb = torch.zeros(cells.shape[0], ld, dtype=torch.float64, device=X.device)
    xq, w = _duffy(2, 3 * order + 2)
    vals, ders = _basis(2, order, xq)
    for q in range(len(w)):
        v, gr = _t(vals[q]), torch.einsum("ckp,ap->cak", Gm, _t(ders[q]))
        u, du = uc @ v, torch.einsum("cja,cak->cjk", uc, gr)     # [cell, comp], [cell, comp, dim]
        wt = vol * float(w[q])
        lap = torch.einsum("cak,cbk,c->cab", gr, gr, wt)
        for c in range(nc):
            L[:, c * nb:(c + 1) * nb, c * nb:(c + 1) * nb] += lap
            lb[:, c * nb:(c + 1) * nb] += (wt * float(D["f"][c]))[:, None] * v
        if nc == 1:
            u0, d0 = u[:, 0], du[:, 0]
            if form == "diffusion":
                a = 1.0 + u0 * u0
                J = a[:, None, None] * gr + 2 * (u0[:, None, None] * v[None, :, None]) * d0[:, None, :]
                Ju = (a + 2 * u0 * u0)[:, None] * d0
            else:
                a = 1.0 + (d0 * d0).sum(dim=1)
                J = a[:, None, None] * gr + 2 * (gr @ d0[:, :, None]) * d0[:, None, :]
                Ju = (a + 2 * (d0 * d0).sum(dim=1))[:, None] * d0
            L += torch.einsum("cjk,cik,c->cji", gr, J, wt)
            lb += torch.einsum("cjk,ck,c->cj", gr, Ju - a[:, None] * d0, wt)
        else:
            adv = torch.einsum("cl,cil->ci", u, gr)              # u . grad phi_i
            conv = torch.einsum("cjl,cl->cj", du, u)             # (u . grad) u
            for c in range(2):
                B = torch.einsum("j,ci,c->cji", v, adv, wt)
                L[:, c * nb:(c + 1) * nb, c * nb:(c + 1) * nb] += B
                for d in range(2):
                    L[:, c * nb:(c + 1) * nb, d * nb:(d + 1) * nb] += torch.einsum("j,i,c->cji", v, v, wt * du[:, c, d])
                lb[:, c * nb:(c + 1) * nb] += (wt * conv[:, c])[:, None] * v     # DG(u) u - G(u) = (u . grad) u
    b = torch.zeros(nc * nd, dtype=torch.float64, device=X.device)
    b.index_add_(0, cdt.reshape(-1), lb.reshape(-1))
    pts = _dof_points(2, order, n)
    fx = _boundary(pts)
    M, b = _eliminate(_csr(cdt, L, nc * nd), b, _t(np.concatenate([fx + c * nd for c in range(nc)])))
    line = _lines(pts, n)
    return _tridiagonal(M, b, torch.cat([line] * nc), spd=False)(b)


def _exact_estimate(case, D):
    dim, order, n = case["dim"], case["order"], case["n"]
    g = _grid(dim, n)
    cells = g.cells.astype(np.int64)
    cd, _, nd = _dofmap(dim, order, 1, n)
    X, ct, cdt = _t(g.coords), _t(cells), _t(cd)
    x0, A, Gm, vol = _geometry(X, ct)
    u = _t(D["u"])
    uc = u[cdt]
    y = torch.zeros(nd, dtype=torch.float64, device=X.device)
    err = torch.zeros(cells.shape[0], dtype=torch.float64, device=X.device)
    xq, w = _duffy(dim, 2)
    _, dv = _basis(dim, order, xq)
    kap = _t(D["kappa"])
    for q in range(len(w)):
        gr = torch.einsum("ckp,ap->cak", Gm, _t(dv[q]))
        du = torch.einsum("ca,cak->ck", uc, gr)
        y.index_add_(0, cdt.reshape(-1), torch.einsum("cak,ck,c->ca", gr, du, vol * kap * float(w[q])).reshape(-1))
        f = _poly(D["terms"], x0 + A @ _t(xq[q]), dim)
        err += ((f - du) ** 2).sum(dim=1) * vol * float(w[q])
    # interior faces: both cells see the same points (weights over the face's vertices, sorted)
    fv, cf = _entities(cells, _FACES[dim])
    nf = fv.shape[0]
    flat = cf.ravel()
    order_ = np.argsort(flat, kind="stable")
    cnt = np.bincount(flat, minlength=nf)
    st = np.concatenate([[0], np.cumsum(cnt)])[:-1]
    inner = np.flatnonzero(cnt == 2)
    c1, c2 = order_[st[inner]] // (dim + 1), order_[st[inner] + 1] // (dim + 1)
    P = g.coords[fv[inner]]
    if dim == 2:
        t = P[:, 1] - P[:, 0]
        nn = np.stack([t[:, 1], -t[:, 0]], axis=1)
    else:
        nn = np.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]) / 2
    area = np.linalg.norm(nn, axis=1)
    nn, ar = _t(nn / area[:, None]), _t(area)
    xq, w = _duffy(dim - 1, 2)
    lam = np.concatenate([1 - xq.sum(axis=1, keepdims=True), xq], axis=1)
    eta = torch.zeros(nf, dtype=torch.float64, device=X.device)
    it = _t(inner)
    c1, c2 = _t(c1), _t(c2)
    for q in range(len(w)):
        xf = _t(np.einsum("fvk,v->fk", P, lam[q]))
        jump, grs = 0, []
        for c, sg in ((c1, 1.0), (c2, -1.0)):
            xh = torch.linalg.solve(A[c], (xf - x0[c])[:, :, None])[:, :, 0]
            gr = torch.einsum("fkp,fap->fak", Gm[c], _basis_at(dim, order, xh)) * sg
            grs.append((c, gr))
            jump = jump + torch.einsum("fa,fak->fk", uc[c], gr)
        for c, gr in grs:
            v = torch.einsum("fak,fk,f->fa", gr, jump, 0.1 * float(w[q]) * ar ** 3)
            y.index_add_(0, cdt[c].reshape(-1), v.reshape(-1))
        eta[it] += (jump * nn).sum(dim=1) ** 2 * float(w[q]) * ar ** 2
    return y, err, eta


def _basis_at(dim, order, x):
    """Reference derivatives at one point per row."""
    dl = _t(np.concatenate([-np.ones((1, dim)), np.eye(dim)]))
    if order == 1:
        return dl.expand(x.shape[0], -1, -1)
    lam = torch.cat([1 - x.sum(dim=1, keepdim=True), x], dim=1)
    d = [(4 * lam[:, i] - 1)[:, None] * dl[i] for i in range(dim + 1)]
    d += [4 * (lam[:, a, None] * dl[b] + lam[:, b, None] * dl[a]) for a, b in _EDGES[dim]]
    return torch.stack(d, dim=1)


def exact(case, seed):
    D = _data(case, seed)
    k = case["kind"]
    if k == "poisson":
        return _exact_poisson(case["dim"], case["order"], case["n"], D["kappa"], 0.0, D["amp"], D["k"])
    if k == "elasticity":
        return _exact_elasticity(case["n"], D["force"])
    if k == "stokes":
        return _exact_stokes(case, D)
    if k == "newton":
        return _exact_newton(case, D)
    if k == "recon":
        if case["target"] in ("RT1", "BDM2"):
            return None
        return _br_rhs(case["dim"], _grid(case["dim"], case["n"]), D["terms"], case["target"])
    if k == "estimate":
        return _exact_estimate(case, D)
    return [_exact_poisson(r["dim"], r["order"], r["n"], r["kappa"], r["alpha"], r["amp"], r["k"]) for r in D["reqs"]]
