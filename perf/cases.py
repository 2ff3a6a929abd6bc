"""Performance cases: the calls a user of this framework makes, from the smallest problem to the
headline's form, each through the public entry points.

A case is a dict of plain values.  ``kind`` says which calls one pass makes:

solve     assembly with new data on a kept operator and a PCG solve (Poisson or elasticity,
          3D hexahedra or 2D quadrilaterals, FP64 or mixed precision, Jacobi or no preconditioner)
tutorial  the tutorial's program: sharp-wave Poisson, unpreconditioned CG, error norms
assemble  assembly with new data, one application of the operator, the right-hand side
bddc      elasticity assembly, BDDC numerical set-up, BDDC-PCG solve
dg        interior-penalty dG assembly and solve
unst      an unstructured hexahedral mesh (random orientation per cell): assembly and solve
batch     one run of a kept plan of independent problems

The symbolic phase (mesh, space, plan) is in ``prepare``: a program with coefficient sweeps, time
steps or a serving loop keeps it, and the framework's own benchmarks call that state "warm".

``exact`` restates the discrete problems in plain torch/numpy in 64 bits: element matrices,
first-visit dof numbering and a CG run down to rounding (for the batch: fast diagonalisation).
"""
import math

import numpy as np
import torch

# Residual tolerances.  They leave the solution with an error well below 1e-9 of the exact discrete
# one: a change of rounding moves CG's iterates, and only the converged solution can be compared.
# 2D and interior-penalty matrices, and CG without a preconditioner, are the worse conditioned.
RTOL, RTOL_TIGHT, RTOL_BATCH = 1e-10, 1e-12, 1e-11
MAXIT = 200000
SHARP3 = [200.0, 0.7, -0.05, -0.05, -0.05]
SHARP2 = [200.0, 0.7, -0.05, -0.05, 0.0]
CLAMP_X0_IDS = [1, 3, 5, 7, 13, 15, 17, 19, 25]  # every n-face of the box on x = 0
NU = 0.3


def listed():
    return [
        # the smallest call: a few hundred dofs, latency and launches; host arrays in and out
        {"name": "poisson_q1_8_fp64", "kind": "solve", "nx": 8, "ny": 8, "nz": 8, "order": 1, "ncomp": 1,
         "precision": "fp64", "host": True},
        # the reference's own CPU-sized case: its first tutorial on 32^3 Q1, FP64 drop-in
        {"name": "tutorial_q1_32", "kind": "tutorial", "nx": 32, "ny": 32, "nz": 32, "order": 1},
        # an ordinary request of a serving loop
        {"name": "poisson_q2_24_mixed", "kind": "solve", "nx": 24, "ny": 24, "nz": 24, "order": 2, "ncomp": 1,
         "precision": "mixed", "host": False},
        # the FP64 drop-in on higher-order elements, odd box
        {"name": "poisson_q3_odd_fp64", "kind": "solve", "nx": 23, "ny": 17, "nz": 21, "order": 3, "ncomp": 1,
         "precision": "fp64", "host": False},
        # the headline's form (Q2, lognormal coefficient, perturbed vertices, mixed precision): the largest
        {"name": "poisson_q2_96_mixed", "kind": "solve", "nx": 96, "ny": 96, "nz": 96, "order": 2, "ncomp": 1,
         "precision": "mixed", "host": False},
        # operator refresh of a program with its own Krylov method (FP64 assembly)
        {"name": "assemble_poisson_q2_64", "kind": "assemble", "nx": 64, "ny": 64, "nz": 64, "order": 2, "ncomp": 1},
        {"name": "assemble_elasticity_q2_32", "kind": "assemble", "nx": 32, "ny": 32, "nz": 32, "order": 2,
         "ncomp": 3},
        # elasticity with jumping coefficients and the BDDC preconditioner on 8^3 subdomains
        {"name": "bddc_elasticity_q2_24", "kind": "bddc", "nx": 24, "ny": 24, "nz": 24, "sub": 8},
        # the tutorial's second formulation (interior penalty)
        {"name": "dg_q2_32_mixed", "kind": "dg", "nx": 32, "ny": 32, "nz": 32, "order": 2, "precision": "mixed"},
        # a mesh from a mesh generator's file: explicit nodes, explicit columns
        {"name": "unstructured_q2_40_mixed", "kind": "unst", "n": 40, "order": 2, "precision": "mixed"},
        # the tutorial's 2D meshes
        {"name": "quad_q2_384_fp64", "kind": "solve", "nx": 384, "ny": 384, "nz": 0, "order": 2, "ncomp": 1,
         "precision": "fp64", "host": False},
        # many small independent problems in one launch
        {"name": "batch_96", "kind": "batch", "count": 96, "nmin": 8, "nmax": 24, "sizes": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, nodes_lo, nodes_hi, order, dim, nmin=2):
    """Cells per direction of a box with about a log-uniform number of nodes, sides apart by up to 1.6."""
    nodes = math.exp(rng.uniform(math.log(nodes_lo), math.log(nodes_hi)))
    side = nodes ** (1.0 / dim) / order
    n = [max(nmin, int(round(side * math.exp(rng.uniform(-0.24, 0.24))))) for _ in range(dim)]
    return n + [0] * (3 - dim)


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "quad", "tutorial", "assemble", "assemble", "bddc", "dg", "unst",
                       "batch"])
    order = rng.choice([1, 2, 2, 3])
    if kind == "solve":
        n = _box(rng, 500, 1500000, order, 3)
        return {"kind": "solve", "nx": n[0], "ny": n[1], "nz": n[2], "order": order, "ncomp": 1,
                "precision": rng.choice(["fp64", "mixed"]), "host": rng.random() < 0.5}
    if kind == "quad":
        n = _box(rng, 500, 600000, order, 2)
        return {"kind": "solve", "nx": n[0], "ny": n[1], "nz": 0, "order": order, "ncomp": 1,
                "precision": rng.choice(["fp64", "mixed"]), "host": rng.random() < 0.5}
    if kind == "tutorial":
        n = _box(rng, 500, 200000, order, 3)
        return {"kind": "tutorial", "nx": n[0], "ny": n[1], "nz": n[2], "order": order}
    if kind == "assemble":
        if rng.random() < 0.5:
            n = _box(rng, 500, 2000000, order, 3)
            return {"kind": "assemble", "nx": n[0], "ny": n[1], "nz": n[2], "order": order, "ncomp": 1}
        n = _box(rng, 500, 270000 if order < 3 else 60000, order, 3)
        return {"kind": "assemble", "nx": n[0], "ny": n[1], "nz": n[2], "order": order, "ncomp": 3}
    if kind == "bddc":
        sub = rng.choice([2, 3, 4])
        n = [rng.randint(2 * sub, 5 * sub) for _ in range(3)]
        return {"kind": "bddc", "nx": n[0], "ny": n[1], "nz": n[2], "sub": sub}
    if kind == "dg":
        n = _box(rng, 500, 150000, order, 3)
        return {"kind": "dg", "nx": n[0], "ny": n[1], "nz": n[2], "order": order,
                "precision": rng.choice(["fp64", "mixed"])}
    if kind == "unst":
        order = rng.choice([1, 2])
        return {"kind": "unst", "n": _log_int(rng, 4, 80 // order), "order": order,
                "precision": rng.choice(["fp64", "mixed"])}
    return {"kind": "batch", "count": _log_int(rng, 4, 96), "nmin": rng.randint(4, 8), "nmax": rng.randint(9, 24),
            "sizes": rng.randint(1, 1 << 20)}


# ---- inputs ---------------------------------------------------------------------------------------------


def _cells_per_dir(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if case.get("nz") else [])


def _vertices(n, rng):
    """Lattice vertices of the unit box (x fastest, 3 coordinates), interior ones moved by up to 0.15 h."""
    dim = len(n)
    ax = [np.arange(k + 1) for k in n]
    ijk = np.stack(np.meshgrid(*ax[::-1], indexing="ij")[::-1], axis=-1).reshape(-1, dim)
    xyz = np.zeros((len(ijk), 3))
    xyz[:, :dim] = ijk / np.array(n)
    inner = np.all((ijk > 0) & (ijk < np.array(n)), axis=1)
    xyz[inner, :dim] += rng.uniform(-0.15, 0.15, size=(int(inner.sum()), dim)) / np.array(n)
    return xyz


def _inputs(case, seed):
    """Vertices, per-cell coefficients and a probe vector's generator, from the seed alone."""
    rng = np.random.Generator(np.random.PCG64([20261203, seed]))
    n = [case["n"]] * 3 if case["kind"] == "unst" else _cells_per_dir(case)
    sigma = 1.5 if (case["kind"] == "bddc" or case.get("ncomp") == 3) else 1.0
    xyz = _vertices(n, rng)
    coef = np.exp(rng.normal(0.0, sigma, size=int(np.prod(n))))
    return n, xyz, coef, rng


def _sizes(case):
    """Cells per direction and order of each problem of a batch, and its coefficient."""
    rng = np.random.Generator(np.random.PCG64([7, case["sizes"]]))
    n = np.round(np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), size=case["count"]))).astype(int)
    p = rng.choice([1, 2, 3], size=case["count"])
    k = rng.uniform(0.1, 10.0, size=case["count"])
    return [(int(a), int(b), float(c)) for a, b, c in zip(n, p, k)]


def _sources(case, seed):
    g = torch.Generator().manual_seed(seed)
    return [torch.randn(n ** 3 * (p + 1) ** 3, dtype=torch.float64, generator=g) for n, p, _ in _sizes(case)]


def _unstructured(case, seed):
    """Cells of the n^3 box with a random orientation each (1-based vertices), and the boundary vefs."""
    from fempar_gb300.bench_unstructured import unstructured_box
    cells, _, ptr, verts, sets = unstructured_box(case["n"], seed=seed)
    return cells, ptr, verts, sets


# ---- one pass -------------------------------------------------------------------------------------------


def _solver(fg, op, precision, precond, rtol=RTOL):
    s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, precond)
    return s.set_parameters_from_pl({"ILS_RTOL": rtol, "ILS_MAX_NUM_ITERATIONS": MAXIT, "PRECISION": precision})


def prepare(case, seed):
    import fempar_gb300 as fg
    ctx = fg.Context(0)
    dev = torch.device("cuda", 0)
    s = {"case": case, "fg": fg, "ctx": ctx}
    kind = case["kind"]
    if kind == "batch":
        from fempar_gb300.batch import BatchSolver
        sizes = _sizes(case)
        lens = [max(p * n - 1, 0) ** 3 for n, p, _ in sizes]
        s["x"] = torch.zeros(sum(lens), dtype=torch.float64, device=dev)
        parts = torch.split(s["x"], lens)
        s["problems"] = [{"n": n, "order": p, "coef": k, "qp_source": f.to(dev), "x": x}
                         for (n, p, k), f, x in zip(sizes, _sources(case, seed), parts)]
        torch.cuda.synchronize()
        s["batch"] = BatchSolver(ctx, s["problems"], rtol=RTOL_BATCH)
        return s
    n, xyz, coef, rng = _inputs(case, seed)
    if kind == "unst":
        cells, ptr, verts, sets = _unstructured(case, seed)
        tri = fg.SerialTriangulation.from_arrays(ctx, xyz, cells, ptr, verts, sets)
    else:
        tri = fg.SerialTriangulation(ctx, n, vertex_xyz=np.ascontiguousarray(xyz.ravel()))
    kdev = torch.from_numpy(coef).to(dev)
    wave = dict(source_fn=fg.FG_FN_SHARP_WAVE, boundary_fn=fg.FG_FN_SHARP_WAVE,
                fn_param=SHARP2 if len(n) == 2 else SHARP3)
    elastic = dict(cell_coef=kdev, nu=NU, source_fn=fg.FG_FN_CONST, fn_param=[0.0, 0.0, -1.0])
    one = dict(source_fn=fg.FG_FN_CONST, fn_param=[1.0])
    mixed = case.get("precision") == "mixed"
    if kind == "dg":
        space = fg.SerialFESpace(tri, order=case["order"], dg=True)
        integ = fg.PoissonIntegration(**wave)
    elif kind == "tutorial":
        space = fg.SerialFESpace(tri, order=case["order"], dirichlet_ids=list(range(1, 27)))
        integ = fg.PoissonIntegration(**wave)
    elif kind == "bddc" or case.get("ncomp") == 3:
        space = fg.SerialFESpace(tri, order=case.get("order", 2), ncomp=3, dirichlet_ids=CLAMP_X0_IDS)
        integ = fg.ElasticityIntegration(**elastic)
    elif kind == "unst":
        space = fg.SerialFESpace(tri, order=case["order"], dirichlet_ids=[1])
        integ = fg.PoissonIntegration(cell_coef=kdev, fast_integration=mixed, **one)
    elif len(n) == 2:
        space = fg.SerialFESpace(tri, order=case["order"], dirichlet_ids=list(range(1, 9)))
        integ = fg.PoissonIntegration(cell_coef=coef if case["host"] else kdev, **wave)
    else:
        space = fg.SerialFESpace(tri, order=case["order"], dirichlet_ids=list(range(1, 27)))
        integ = fg.PoissonIntegration(cell_coef=coef if case.get("host") else kdev, fast_integration=mixed, **one)
    op = fg.FEAffineOperator(space, integ).compute()
    s["op"] = op
    if kind == "assemble":
        s["x"] = torch.from_numpy(rng.standard_normal(space.num_free_dofs)).to(dev)
        s["y"] = torch.empty_like(s["x"])
    elif kind == "bddc":
        s["bddc"] = fg.MLBDDC(op, nsub=(case["sub"],) * 3, use_faces=True, weighting=fg.FG_BDDC_WEIGHT_STIFFNESS)
        s["solver"] = _solver(fg, op, "mixed", s["bddc"])
    else:
        s["solver"] = _solver(fg, op, case.get("precision", "fp64"), "identity" if kind == "tutorial" else "jacobi",
                              RTOL_TIGHT if kind in ("tutorial", "dg") or len(n) == 2 else RTOL)
    if kind in ("bddc", "dg", "unst", "solve"):
        s["x"] = torch.empty(space.num_free_dofs, dtype=torch.float64, device=dev)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].run()
        return state["x"]
    op = state["op"].compute()
    if kind == "assemble":
        op.apply_device(state["x"], state["y"])
        return {"y": state["y"], "rhs": op.get_translation()}
    if kind == "tutorial":
        x = state["solver"].solve()
        return {"x": x, "norms": op.error_norms(x, state["fg"].FG_FN_SHARP_WAVE, SHARP3)}
    if kind == "bddc":
        state["bddc"].numerical_setup()
    if case.get("host"):
        return state["solver"].solve()
    return state["solver"].solve_device(x=state["x"])


# ---- what a pass cannot do without ----------------------------------------------------------------------


def _space_counts(n, order, ncomp, dg=False):
    """Free rows (about) and nonzeros of the matrix of a box."""
    if dg:
        nn = (order + 1) ** 3
        cells = n[0] * n[1] * n[2]
        return cells * nn, cells * nn * nn * 7
    rows = nnz = 1.0
    for k in n:
        rows *= order * k - 1 if ncomp == 1 else order * k
        nnz *= k * (order + 1) ** 2 - k  # one direction's mass-matrix entries
    return rows * ncomp, nnz * ncomp ** 2


def work(case):
    """Bytes and flops of one pass: element integrals once, the coefficients and vertices read, the
    matrix written once, and for a solve each iteration's read of the matrix; the number of
    iterations is the usual growth with the nodes per direction."""
    kind = case["kind"]
    if kind == "batch":
        nbytes = flops = 0.0
        for n, p, _ in _sizes(case):
            rows, nnz = _space_counts([n] * 3, p, 1)
            nbytes += 8.0 * (n ** 3 * (p + 1) ** 3 + rows)
            flops += 2.0 * nnz * 4 * p * n
        return {"bytes": nbytes, "flops": flops}
    n = [case["n"]] * 3 if kind == "unst" else _cells_per_dir(case)
    dim = len(n)
    order = case.get("order", 2)
    ncomp = 3 if kind == "bddc" else case.get("ncomp", 1)
    rows, nnz = _space_counts(n, order, ncomp, dg=kind == "dg")
    cells = float(np.prod(n))
    nd = (order + 1) ** dim
    nbytes = 8.0 * (cells + 3 * cells + nnz + rows)
    flops = float(cells * nd * (nd + 1) * nd * dim * (1 if ncomp == 1 else 3))
    its = 0.0
    if kind in ("solve", "unst", "dg"):
        its = 5.0 * order * max(n)
    elif kind == "tutorial":
        its = 3.0 * order * max(n)
    elif kind == "assemble":
        its = 1.0
    elif kind == "bddc":
        its = 50.0
        local = 3.0 * float(np.prod([order * k / case["sub"] + 1 for k in n]))
        flops += case["sub"] ** 3 * local ** 3 / 3.0
    width = 4.0 if case.get("precision") == "mixed" else 8.0
    return {"bytes": nbytes + its * (nnz * width + 2 * rows * width), "flops": flops + its * 2.0 * nnz}


# ---- the same results in plain torch / numpy, 64 bits ---------------------------------------------------


def _device():
    return torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")


def _lagrange(p, x):
    """Values and derivatives of the equispaced Lagrange basis of order p on [-1, 1] at points x."""
    nodes = np.linspace(-1.0, 1.0, p + 1)
    val = np.ones((p + 1, len(x)))
    der = np.zeros((p + 1, len(x)))
    for j in range(p + 1):
        for k in range(p + 1):
            if k != j:
                f = (x - nodes[k]) / (nodes[j] - nodes[k])
                der[j] = der[j] * f + val[j] / (nodes[j] - nodes[k])
                val[j] = val[j] * f
    return val, der


def _tensor(tabs):
    """Outer product of per-direction tables (nodes, points), x fastest in both."""
    out = np.ones((1, 1))
    for t in tabs:
        out = np.einsum("aq,bp->bapq", out, t).reshape(t.shape[0] * out.shape[0], -1)
    return out


def _tables(p, points):
    """Shape values (nodes, points) and gradients (nodes, points, dim) at a tensor set of points, one
    array of coordinates per direction."""
    dim = len(points)
    vd = [_lagrange(p, x) for x in points]
    shp = _tensor([v for v, _ in vd])
    grad = np.stack([_tensor([vd[d][1] if d == j else vd[d][0] for d in range(dim)]) for j in range(dim)], axis=-1)
    return shp, grad


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_device())


def _jacobian(xv, ggrad):
    """J[c, q, i, j] = d x_i / d xi_j."""
    return torch.einsum("cki,kqj->cqij", xv, ggrad)


def _wave(x, prm, dim):
    """u and f = -lap u of the sharp wave at x (..., 3)."""
    alpha, r = prm[0], prm[1]
    rho = (x[..., :dim] - torch.as_tensor(prm[2:2 + dim], dtype=x.dtype, device=x.device)).norm(dim=-1)
    t = rho - r
    a = 1.0 + (alpha * t) ** 2
    lap = -2.0 * alpha ** 3 * t / a ** 2 + (dim - 1) / rho * alpha / a
    return torch.atan(alpha * t), -lap


def _nface_nodes(p, dim):
    """Local nodes of the cell's interior, then of each n-face in (dimension, code) order."""
    faces = [(a | (t << dim), bin(t).count("1")) for t in range(1 << dim) for a in range(1 << dim) if not a & t]
    faces.sort(key=lambda f: (f[1], f[0]))
    lists = []
    for code, _ in [faces[-1]] + faces[:-1]:
        a, t = code & ((1 << dim) - 1), code >> dim
        ranges = [range(1, p) if (t >> d) & 1 else [p * ((a >> d) & 1)] for d in range(dim)]
        nodes = [0]
        for d in range(dim - 1, -1, -1):
            nodes = [m + i * (p + 1) ** d for m in nodes for i in ranges[d]]
        lists.append(nodes)
    return lists


def _cell_lattice(n):
    """(cells, 2^dim) lattice coordinates of the cells' vertices of a box, (cells, 2^dim, dim)."""
    dim = len(n)
    ax = [np.arange(k) for k in n]
    c = np.stack(np.meshgrid(*ax[::-1], indexing="ij")[::-1], axis=-1).reshape(-1, 1, dim)
    b = np.array([[(v >> d) & 1 for d in range(dim)] for v in range(1 << dim)])
    return c + b


class _Discrete:
    """Element matrices E, element vectors, 0-based free dof ids per cell (n for Dirichlet dofs)."""

    def __init__(self, case, seed):
        kind = case["kind"]
        p = case.get("order", 2)
        n, xyz, coef, rng = _inputs(case, seed)
        dim = len(n)
        nc = 3 if (kind == "bddc" or case.get("ncomp") == 3) else 1
        if kind == "unst":
            cv = _unstructured(case, seed)[0].astype(np.int64) - 1
            m = case["n"] + 1
            lat = np.stack([cv % m, (cv // m) % m, cv // (m * m)], axis=-1)
        else:
            lat = _cell_lattice(n)
            stride = np.cumprod([1] + [k + 1 for k in n[:-1]])
            cv = lat @ stride
        self.rng = rng
        xv = _t(xyz[:, :dim])[torch.as_tensor(cv, device=_device())]
        gx, gw = np.polynomial.legendre.leggauss(p + 1)
        shp, grad = _tables(p, [gx] * dim)
        w = _tensor([gw[None, :]] * dim)[0]
        gshp, ggrad = _tables(1, [gx] * dim)
        # lattice position of every local node: the corners' multilinear combination, times p
        nodes1 = np.linspace(-1.0, 1.0, p + 1)
        corner = _tables(1, [nodes1] * dim)[0]
        pos = np.rint(np.einsum("ckd,ka->cad", p * lat.astype(float), corner)).astype(np.int64)
        full = np.array([p * k + 1 for k in n])
        key = pos @ np.cumprod(np.concatenate([[1], full[:-1]]))
        wall = (pos == 0) | (pos == full - 1)
        fixed = wall[..., 0] & (pos[..., 0] == 0) if nc == 3 else wall.any(axis=-1)
        nn = key.shape[1]
        # first-visit numbering: cell by cell, interior then n-faces, component by component
        visit = [(a, c) for nodes in _nface_nodes(p, dim) for c in range(nc) for a in nodes]
        va, vc = np.array([v[0] for v in visit]), np.array([v[1] for v in visit])
        seq = key[:, va] * nc + vc
        seq = seq[~fixed[:, va]]
        ids, first = np.unique(seq, return_index=True)
        rank = np.empty(len(ids), dtype=np.int64)
        rank[np.argsort(first)] = np.arange(len(ids))
        self.n = len(ids)
        allkeys = (key[:, None, :] * nc + np.arange(nc)[None, :, None]).reshape(len(key), -1)
        allfix = np.repeat(fixed[:, None, :], nc, axis=1).reshape(len(key), -1)
        at = np.minimum(np.searchsorted(ids, allkeys), max(len(ids) - 1, 0))
        self.gid = torch.as_tensor(np.where(allfix, self.n, rank[at]), device=_device())
        # element matrices and vectors, a chunk of cells at a time
        grad, ggrad, gshp, w, shp = _t(grad), _t(ggrad), _t(gshp), _t(w), _t(shp)
        wave = kind in ("tutorial",) or dim == 2
        prm = SHARP2 if dim == 2 else SHARP3
        k = _t(np.ones_like(coef) if kind == "tutorial" else coef)
        nodex = torch.einsum("cki,ka->cai", xv, _t(corner))
        gval = _wave(nodex, prm, dim)[0] if wave else None
        self.E, rhs = [], torch.zeros(self.n + 1, dtype=torch.float64, device=_device())
        step = max(1, int(2e8 // (nn * nn * dim)))
        for c0 in range(0, len(cv), step):
            sl = slice(c0, c0 + step)
            J = _jacobian(xv[sl], ggrad)
            det = torch.linalg.det(J)
            det = torch.where(det[:, :1] < 0, det.abs(), det)
            # s_a = J^-T grad_ref
            G = torch.einsum("aqj,cqji->cqai", grad, torch.linalg.inv(J))
            fac = det * w
            if nc == 1:
                S = G * (fac * k[sl, None]).sqrt()[..., None, None]
                S = S.permute(0, 2, 1, 3).reshape(len(S), nn, -1)
                E = S @ S.transpose(1, 2)
                f = _wave(torch.einsum("cki,kq->cqi", xv[sl], gshp), prm, dim)[1] if wave else torch.ones_like(fac)
                ev = torch.einsum("cq,aq->ca", fac * f, shp)
            else:
                S = (G * fac.sqrt()[..., None, None]).permute(0, 3, 2, 1).reshape(len(G), 3 * nn, -1)
                A = (S @ S.transpose(1, 2)).reshape(-1, 3, nn, 3, nn)
                lam = (NU * k[sl] / ((1 + NU) * (1 - 2 * NU)))[:, None, None, None, None]
                mu = (k[sl] / (2 * (1 + NU)))[:, None, None, None, None]
                E = lam * A + mu * A.permute(0, 3, 2, 1, 4)
                tr = A[:, 0, :, 0] + A[:, 1, :, 1] + A[:, 2, :, 2]
                for d in range(3):
                    E[:, d, :, d] += mu[:, 0, 0] * tr
                E = E.reshape(-1, 3 * nn, 3 * nn)
                ev = torch.zeros(len(E), 3, nn, dtype=torch.float64, device=_device())
                ev[:, 2] = -torch.einsum("cq,aq->ca", fac, shp)
                ev = ev.reshape(len(E), -1)
            if gval is not None:
                fx = torch.where(self.gid[sl] == self.n, gval[sl], torch.zeros_like(gval[sl]))
                ev = ev - torch.einsum("cab,cb->ca", E, fx)
            rhs.index_add_(0, self.gid[sl].reshape(-1), ev.reshape(-1))
            self.E.append(E)
        self.step = step
        self.b = rhs[:self.n]

    def apply(self, x):
        xp = torch.cat([x, x.new_zeros(1)])
        y = torch.zeros_like(xp)
        for i, E in enumerate(self.E):
            g = self.gid[i * self.step:(i + 1) * self.step]
            y.index_add_(0, g.reshape(-1), torch.bmm(E, xp[g][..., None]).reshape(-1))
        return y[:self.n]

    def diagonal(self):
        d = torch.zeros(self.n + 1, dtype=torch.float64, device=_device())
        for i, E in enumerate(self.E):
            d.index_add_(0, self.gid[i * self.step:(i + 1) * self.step].reshape(-1),
                         torch.diagonal(E, dim1=1, dim2=2).reshape(-1))
        return d[:self.n]


class _DiscreteDG:
    """Interior penalty on a structured box, k = 1, weak sharp-wave data: cell blocks and, per
    direction, the blocks of the facets between neighbours."""

    def __init__(self, case, seed):
        p = case["order"]
        n, xyz, _, _ = _inputs(case, seed)
        lat = _cell_lattice(n)
        cv = lat @ np.cumprod([1, n[0] + 1, n[1] + 1])
        xv = _t(xyz)[torch.as_tensor(cv, device=_device())]
        gx, gw = np.polynomial.legendre.leggauss(p + 1)
        shp, grad = (_t(a) for a in _tables(p, [gx] * 3))
        gshp, ggrad = (_t(a) for a in _tables(1, [gx] * 3))
        w = _t(_tensor([gw[None, :]] * 3)[0])
        J = _jacobian(xv, ggrad)
        det = torch.linalg.det(J)
        S = torch.einsum("aqj,cqji->caqi", grad, torch.linalg.inv(J)) * (det * w).sqrt()[:, None, :, None]
        S = S.reshape(len(S), S.shape[1], -1)
        self.D = S @ S.transpose(1, 2)
        f = _wave(torch.einsum("cki,kq->cqi", xv, gshp), SHARP3, 3)[1]
        self.b = torch.einsum("cq,aq->ca", det * w * f, shp)
        del S, J
        self.nc, self.nn = self.b.shape
        self.links = []
        wf = _t(_tensor([gw[None, :]] * 2)[0])
        ids = torch.arange(self.nc, device=_device()).reshape(n[2], n[1], n[0])
        cip = 10.0 * p * p

        def side(cells, d, s):
            """Shapes, normal derivatives with n = +d direction's unit normal, area weights, h, points."""
            pts = [np.array([s]) if e == d else gx for e in range(3)]
            v, g = (_t(a) for a in _tables(p, pts))
            gv, gg = (_t(a) for a in _tables(1, pts))
            Jf = _jacobian(xv[cells], gg)
            Ji = torch.linalg.inv(Jf)
            h = 2.0 * (1.0 / Ji.norm(dim=-1).prod(dim=-1)) ** (1.0 / 3.0)
            t1, t2 = [e for e in range(3) if e != d]
            nrm = torch.linalg.cross(Jf[..., t1], Jf[..., t2])
            nrm = nrm if d != 1 else -nrm
            area = nrm.norm(dim=-1)
            nrm = nrm / area[..., None] * torch.sign(torch.linalg.det(Jf))[:, :1, None]
            dn = torch.einsum("aqj,cqji,cqi->caq", g, Ji, nrm)
            return v, dn, area * wf, h, torch.einsum("cki,kq->cqi", xv[cells], gv)

        for d in range(3):
            ax = 2 - d
            last = ids.shape[ax] - 1
            lo = ids.narrow(ax, 0, last).reshape(-1)
            hi = ids.narrow(ax, 1, last).reshape(-1)
            if len(lo):
                vl, dl, al, hl, _ = side(lo, d, 1.0)
                vr, dr, _, hr, _ = side(hi, d, -1.0)
                pen = cip / torch.minimum(hl, hr) * al
                V = [vl.expand(len(lo), -1, -1), vr.expand(len(lo), -1, -1)]
                N = [dl, -dr]  # grad . n_I
                B = {}
                for i in (0, 1):
                    for j in (0, 1):
                        # n_i . n_j = 1 or -1, and grad phi_j . n_i is that times grad phi_j . n_j
                        sg = 1.0 if i == j else -1.0
                        B[i, j] = -sg * (0.5 * (al[:, None] * V[i]) @ N[j].transpose(1, 2)
                                         + 0.5 * (al[:, None] * N[i]) @ V[j].transpose(1, 2)
                                         - (pen[:, None] * V[i]) @ V[j].transpose(1, 2))
                self.D.index_add_(0, lo, B[0, 0])
                self.D.index_add_(0, hi, B[1, 1])
                self.links.append((lo, hi, B[0, 1], B[1, 0]))
            for cells, s in ((ids.select(ax, 0).reshape(-1), -1.0), (ids.select(ax, last).reshape(-1), 1.0)):
                v, dn, a, h, x = side(cells, d, s)
                dn = dn * s
                v = v.expand(len(cells), -1, -1)
                pen = cip / h * a
                wa = a[:, None] * v
                blk = -(wa @ dn.transpose(1, 2)) - (dn @ wa.transpose(1, 2)) + (pen[:, None] * v) @ v.transpose(1, 2)
                self.D.index_add_(0, cells, blk)
                g = _wave(x, SHARP3, 3)[0]
                self.b.index_add_(0, cells, -torch.einsum("caq,cq->ca", dn, a * g)
                                  + torch.einsum("caq,cq->ca", v, pen * g))
        self.b = self.b.reshape(-1)
        self.n = len(self.b)

    def apply(self, x):
        x = x.reshape(self.nc, self.nn, 1)
        y = torch.bmm(self.D, x)
        for lo, hi, lr, rl in self.links:
            y.index_add_(0, lo, torch.bmm(lr, x[hi]))
            y.index_add_(0, hi, torch.bmm(rl, x[lo]))
        return y.reshape(-1)

    def diagonal(self):
        return torch.diagonal(self.D, dim1=1, dim2=2).reshape(-1).clone()


def _solve(A, jacobi=True):
    """CG on A x = b down to rounding (the true residual is refreshed and the run repeated once)."""
    m = 1.0 / A.diagonal() if jacobi else torch.ones_like(A.b)
    x = torch.zeros_like(A.b)
    for _ in range(2):
        r = A.b - A.apply(x)
        stop = 1e-13 * A.b.norm()
        if r.norm() <= stop:
            break
        z = m * r
        p = z.clone()
        rz = torch.dot(r, z)
        for it in range(1, 100000):
            q = A.apply(p)
            alpha = rz / torch.dot(p, q)
            x += alpha * p
            r -= alpha * q
            z = m * r
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
            if it % 25 == 0 and r.norm() <= stop:
                break
    return x


def _batch_exact(case, seed):
    """Fast diagonalisation: the uniform-cell operator is a sum of products of 1D mass and stiffness."""
    out = []
    for (n, p, k), f in zip(_sizes(case), _sources(case, seed)):
        q = p + 1
        gx, gw = np.polynomial.legendre.leggauss(q)
        v, dv = _lagrange(p, gx)
        h = 1.0 / n
        me, ke = (v * gw) @ v.T * (h / 2), (dv * gw) @ dv.T * (2 / h)
        N = p * n + 1
        M, K, L = np.zeros((N, N)), np.zeros((N, N)), np.zeros((N, n * q))
        for c in range(n):
            s = slice(p * c, p * c + q)
            M[s, s] += me
            K[s, s] += ke
            L[s, c * q:(c + 1) * q] = v * gw * (h / 2)
        M, K, L = M[1:-1, 1:-1], K[1:-1, 1:-1], L[1:-1]
        C = np.linalg.cholesky(M)
        Ci = np.linalg.inv(C)
        lam, U = np.linalg.eigh(Ci @ K @ Ci.T)
        T = Ci.T @ U  # T^T M T = I, T^T K T = diag(lam)
        F = f.numpy().reshape(n, n, n, q, q, q).transpose(0, 3, 1, 4, 2, 5).reshape(n * q, n * q, n * q)
        W = T.T @ L
        b = np.einsum("zyx,kz,jy,ix->kji", F, W, W, W, optimize=True)
        u = b / (k * (lam[:, None, None] + lam[None, :, None] + lam[None, None, :]))
        out.append(np.einsum("kji,zk,yj,xi->zyx", u, T, T, T, optimize=True).ravel())
    return np.concatenate(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _batch_exact(case, seed)
    if kind == "dg":
        return _solve(_DiscreteDG(case, seed))
    A = _Discrete(case, seed)
    if kind == "assemble":
        return {"y": A.apply(_t(A.rng.standard_normal(A.n))), "rhs": A.b.cpu().numpy()}
    x = _solve(A, jacobi=kind != "tutorial")
    if kind == "tutorial":
        return {"x": x.cpu().numpy(), "norms": None}
    return x.cpu().numpy() if case.get("host") else x
