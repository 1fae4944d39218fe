"""The calls whose speed this library is judged by, at the sizes that programs use.

An operator is set up once by a program and applied to many vectors (a Krylov
solver, a time loop), a multigrid hierarchy likewise, and a network is trained
over many batches: the handles are made once per size and kept, the vectors
and samples of a call come from the seed.  Meshes are the jittered Kuhn boxes
that the benchmark and the tests use, or the same cells with shuffled
numbering read as an unstructured mesh.

exact() restates every linear call in 64 bits with plain torch, from the mesh
arrays: reference integrals of the Lagrange basis from its monomials, face
integrals by Gauss quadrature.
"""
import functools
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "simplex-benchmarks_b200"))
import simplexfem as sf  # noqa: E402

MASS = 1e5  # mass coefficient of the Helmholtz operator (the library's default)
# a batch of many small problems: 8 .. 8 + n hexes per direction, as in the benchmark
BATCH_BASE = 8


def _vmult(name, kind, degree, precision, n, components=1, mesh="box"):
    return {"name": name, "call": "vmult", "kind": kind, "degree": degree, "precision": precision,
            "components": components, "mesh": mesh, "nx": n[0], "ny": n[1], "nz": n[2]}


def listed():
    return [
        # The smallest operator application in use: a coarse level or a test
        # problem, where launches and host work decide.
        _vmult("cg_p2_f64_16", "cg", 2, "fp64", (16, 16, 16)),
        # The largest Poisson operator of the benchmark (17M unknowns).
        _vmult("cg_p2_f64_128", "cg", 2, "fp64", (128, 128, 128)),
        # The finest level of the mixed-precision multigrid: FP32 smoothing and residuals.
        _vmult("cg_p3_f32_64", "cg", 3, "fp32", (64, 64, 64)),
        # A box whose sides no tile divides.
        _vmult("cg_p3_f64_odd", "cg", 3, "fp64", (37, 41, 35)),
        # A mesh from a file: arbitrary vertex and cell numbering.
        _vmult("cg_p2_f64_arrays", "cg", 2, "fp64", (44, 40, 36), mesh="arrays"),
        # Three-component Laplace (displacements, velocities).
        _vmult("cg_vec_p2_f64_48", "cg", 2, "fp64", (48, 48, 48), components=3),
        # The headline workload: DG SIPG P3, 3.9M unknowns.
        _vmult("dg_p3_f64_32", "dg", 3, "fp64", (32, 32, 32)),
        # DG of lower degree in FP32 (a level of a DG hierarchy), odd sides.
        _vmult("dg_p2_f32_odd", "dg", 2, "fp32", (45, 38, 31)),
        # Many Helmholtz problems of different sizes in one launch (one per lung
        # generation in the reference): 110M unknowns.
        {"name": "helmholtz_batch_p2_f64", "call": "batch", "degree": 2, "precision": "fp64", "problems": 32},
        # The Poisson solve of the benchmark: mixed multigrid-preconditioned CG to 1e-8.
        {"name": "solve_cg_p3_64", "call": "solve", "kind": "cg", "degree": 3, "n": 64, "levels": "fp32"},
        # The same solver on DG: DG smoothing on top of the continuous hierarchy.
        {"name": "solve_dg_p3_16", "call": "solve", "kind": "dg", "degree": 3, "n": 16, "levels": "fp32"},
        # One backward pass of the learned smoother's training: a batch of the default size.
        {"name": "mlp_gradient_2048", "call": "mlp", "samples": 2048},
    ]


def draw(rng):
    """One more case: mostly operator applications over degrees, precisions,
    sizes and meshes, some batches, solves and training batches."""
    pick = rng.random()
    if pick < 0.1:
        return {"call": "batch", "degree": rng.choice([1, 2, 3]), "precision": rng.choice(["fp64", "fp32"]),
                "problems": rng.randint(2, 16)}
    if pick < 0.2:
        kind = rng.choice(["cg", "cg", "dg"])
        return {"call": "solve", "kind": kind, "degree": rng.choice([2, 3]), "n": rng.choice([8, 16, 32]),
                "levels": rng.choice(["fp32", "fp64"])}
    if pick < 0.28:
        return {"call": "mlp", "samples": int(2 ** rng.uniform(8, 15))}
    kind = rng.choice(["cg", "cg", "dg", "helmholtz"])
    components = 3 if kind == "helmholtz" or (kind == "cg" and rng.random() < 0.25) else 1
    degree = rng.choice([1, 2, 2, 3, 3])
    mesh = "arrays" if rng.random() < 0.2 else "box"
    top = {1: 80, 2: 64, 3: 48}[degree] if components == 1 else {1: 56, 2: 44, 3: 32}[degree]
    n = int(round(math.exp(rng.uniform(math.log(4), math.log(top)))))
    if rng.random() < 0.4:
        sides = [4 * max(1, n // 4)] * 3
    else:
        sides = [max(2, int(n * rng.uniform(0.75, 1.25))) for _ in range(3)]
    c = _vmult("", kind, degree, rng.choice(["fp64", "fp64", "fp32"]), sides, components, mesh)
    del c["name"]
    return c


# ---- what a program keeps ------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _mesh(how, nx, ny, nz, jitter=0.1):
    box = sf.Mesh((nx, ny, nz), jitter=jitter, seed=0)
    if how == "box":
        return box
    rng = np.random.default_rng(7)
    x, cells = box.vertices(), box.cells()
    relabel = rng.permutation(len(x))
    y = np.empty_like(x)
    y[relabel] = x
    return sf.Mesh.from_arrays(y, rng.permuted(relabel[cells[rng.permutation(len(cells))]], axis=1))


@functools.lru_cache(maxsize=None)
def _operator(kind, degree, precision, components, how, nx, ny, nz):
    return sf.Operator(_mesh(how, nx, ny, nz), degree, kind, precision, n_components=components)


def _operator_of(case):
    return _operator(*(case[k] for k in ("kind", "degree", "precision", "components", "mesh", "nx", "ny", "nz")))


def _batch_sizes(problems):
    return [BATCH_BASE + problems * i // max(1, problems - 1) for i in range(problems)]


@functools.lru_cache(maxsize=None)
def _batch(degree, precision, problems):
    return sf.Batch([_operator("helmholtz", degree, precision, 3, "box", n, n, n) for n in _batch_sizes(problems)])


@functools.lru_cache(maxsize=None)
def _solver(kind, degree, n, levels):
    op = sf.Operator(_mesh("box", n, n, n, 0.0), degree, kind, "fp64")
    # DG: the continuous space of the same degree right below (c_transfer 1)
    mg = sf.Multigrid(op, precision=levels, c_transfer=1 if kind == "dg" else 0)
    return op, sf.SolverCG(op, mg)


def _values(op, seed, k=0):
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + k)
    return torch.rand(op.m(), generator=g, dtype=op.dtype, device="cuda") * 2 - 1


def prepare(case, seed):
    call = case["call"]
    if call == "vmult":
        op = _operator_of(case)
        return {"call": call, "op": op, "src": _values(op, seed), "dst": op.initialize_dof_vector()}
    if call == "batch":
        b = _batch(case["degree"], case["precision"], case["problems"])
        return {"call": call, "batch": b, "src": [_values(o, seed, k) for k, o in enumerate(b.ops)],
                "dst": [o.initialize_dof_vector() for o in b.ops]}
    if call == "solve":
        op, cg = _solver(case["kind"], case["degree"], case["n"], case["levels"])
        return {"call": call, "op": op, "cg": cg, "b": sf.rhs(op, sf.sine_modes_rhs(seed=seed)),
                "x": op.initialize_dof_vector()}
    # samples as the training makes them: residuals of unit norm, the cell's
    # scaled Jacobian, and errors of the residual's size
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["samples"]
    r = torch.randn(n, 20, generator=g, device="cuda")
    r /= r.norm(dim=1, keepdim=True)
    j = torch.eye(3, device="cuda").reshape(1, 9) + 0.3 * torch.randn(n, 9, generator=g, device="cuda")
    y = 0.3 * r + 0.1 * torch.randn(n, 20, generator=g, device="cuda")
    return {"call": call, "mlp": sf.MLP(seed=1), "X": torch.cat([r, j], 1).contiguous(), "Y": y}


def run(state):
    call = state["call"]
    if call == "vmult":
        state["op"].vmult(state["dst"], state["src"])
        return state["dst"]
    if call == "batch":
        state["batch"].vmult(state["dst"], state["src"])
        return state["dst"]
    if call == "solve":
        state["x"].zero_()
        state["cg"].solve(state["x"], state["b"], rtol=1e-8)
        return state["x"]
    return state["mlp"].gradient(state["X"], state["Y"])


# ---- reference element -----------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _nodes(p):
    """Barycentric multi-indices of the P_p nodes: vertices, edges from the
    lower to the higher vertex, faces opposite vertex 0 .. 3."""
    def unit(*parts):
        a = [0, 0, 0, 0]
        for v, k in parts:
            a[v] += k
        return tuple(a)

    out = [unit((v, p)) for v in range(4)]
    for i, j in itertools.combinations(range(4), 2):
        out += [unit((i, p - k), (j, k)) for k in range(1, p)]
    if p == 3:
        out += [unit(*[(v, 1) for v in range(4) if v != f]) for f in range(4)]
    return out


@functools.lru_cache(maxsize=None)
def _monomials(p):
    e = [m for m in itertools.product(range(p + 1), repeat=3) if sum(m) <= p]
    v = np.array([[np.prod([(a[d + 1] / p) ** m[d] for d in range(3)]) for m in e] for a in _nodes(p)])
    return e, np.linalg.inv(v)  # column i: coefficients of basis function i


def _basis(p, xi):
    """Values [q][K] and gradients [q][K][3] of the P_p basis at points xi."""
    e, c = _monomials(p)
    power = lambda x, k: x ** k if k > 0 else np.ones_like(x)  # noqa: E731
    v = np.stack([np.prod([power(xi[:, d], m[d]) for d in range(3)], axis=0) for m in e], 1)
    g = np.zeros((len(xi), len(e), 3))
    for k, m in enumerate(e):
        for d in range(3):
            if m[d]:
                g[:, k, d] = m[d] * np.prod([power(xi[:, a], m[a] - (a == d)) for a in range(3)], axis=0)
    return v @ c, np.einsum("qmd,mi->qid", g, c)


@functools.lru_cache(maxsize=None)
def _gauss(n):
    t, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (t + 1), 0.5 * w


@functools.lru_cache(maxsize=None)
def _cell_matrices(p):
    """Reference stiffness [3][3][K][K] and mass [K][K]."""
    t, w = _gauss(p + 2)
    pts, wts = [], []
    for (a, wa), (b, wb), (c, wc) in itertools.product(zip(t, w), repeat=3):
        pts.append((a, b * (1 - a), c * (1 - a) * (1 - b)))
        wts.append(wa * wb * wc * (1 - a) ** 2 * (1 - b))
    v, g = _basis(p, np.array(pts))
    wts = np.array(wts)
    return np.einsum("q,qia,qjb->abij", wts, g, g), np.einsum("q,qi,qj->ij", wts, v, v)


@functools.lru_cache(maxsize=None)
def _face_points(p):
    """Weights (sum 1) and, per face, values [q][K] and gradients [q][K][3] at
    the same points seen from either side: a cell's vertices ascend globally."""
    t, w = _gauss(p + 2)
    lam, wts = [], []
    for (a, wa), (b, wb) in itertools.product(zip(t, w), repeat=2):
        lam.append((1 - a - b * (1 - a), a, b * (1 - a)))
        wts.append(2 * wa * wb * (1 - a))
    lam = np.array(lam)
    faces = []
    for f in range(4):
        bary = np.zeros((len(lam), 4))
        bary[:, [v for v in range(4) if v != f]] = lam
        faces.append(_basis(p, bary[:, 1:]))
    return np.array(wts), faces


# ---- the operators in 64 bits ------------------------------------------------------------------


def _geometry(mesh):
    x = torch.from_numpy(mesh.vertices()).cuda()
    c = torch.from_numpy(mesh.cells().astype(np.int64)).cuda()
    v = x[c]
    jac = (v[:, 1:] - v[:, :1]).transpose(1, 2).contiguous()
    return v, torch.linalg.inv(jac), torch.linalg.det(jac).abs()


def _tensor(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def _laplace(p, jinv, det, u):
    """Cell Laplace of u [cells][components][K]."""
    s = _tensor(_cell_matrices(p)[0])
    g = torch.einsum("cad,cbd->cab", jinv, jinv) * det[:, None, None]
    y = torch.zeros_like(u)
    for a in range(3):
        for b in range(3):
            y += g[:, a, b][:, None, None] * (u @ s[a, b].T)
    return y


def _exact_cg(mesh, p, components, src):
    dofs, fixed = mesh.cg_dofs(p)
    dofs = torch.from_numpy(dofs.astype(np.int64)).cuda()
    fixed = torch.from_numpy(fixed.astype(bool)).cuda()
    _, jinv, det = _geometry(mesh)
    x = src.double().reshape(-1, components)
    x0 = torch.where(fixed[:, None], torch.zeros_like(x), x)
    y = torch.zeros_like(x)
    for a in range(0, len(dofs), 1 << 19):
        d = dofs[a:a + (1 << 19)]
        z = _laplace(p, jinv[a:a + len(d)], det[a:a + len(d)], x0[d].transpose(1, 2))
        y.index_add_(0, d.reshape(-1), z.transpose(1, 2).reshape(-1, components))
    return torch.where(fixed[:, None], x, y).reshape(-1)


def _exact_dg(mesh, p, components, helmholtz, src):
    nb, nbf = (torch.from_numpy(a.astype(np.int64)).cuda() for a in mesh.neighbors())
    v, jinv, det = _geometry(mesh)
    u = src.double().reshape(len(v), components, -1)
    w, faces = _face_points(p)
    w = _tensor(w)
    phi = [_tensor(f[0]) for f in faces]
    dphi = [_tensor(f[1]) for f in faces]
    area, normal = [], []
    for f in range(4):
        a, b, c = (v[:, k] for k in range(4) if k != f)
        n = torch.linalg.cross(b - a, c - a)
        size = n.norm(dim=1)
        n = n / size[:, None]
        out = ((a - v[:, f]) * n).sum(1).sign()
        area.append(0.5 * size)
        normal.append(n * out[:, None])
    factor = (p + 1) * (p + 3) / 3
    if helmholtz:
        inv_h = torch.stack([2 * a / det for a in area], 1)
    else:
        inside = torch.where(nb >= 0, 0.5, 1.0)
        tau = (torch.stack(area, 1) * inside).sum(1) / (det / 6)
    y = _laplace(p, jinv, det, u)
    if helmholtz:
        y += MASS * det[:, None, None] * (u @ _tensor(_cell_matrices(p)[1]).T)
    for f in range(4):
        for a in range(0, len(v), 1 << 16):
            e = slice(a, min(len(v), a + (1 << 16)))
            n = normal[f][e]
            own_n = torch.einsum("cad,cd->ca", jinv[e], n)
            other, of = nb[e, f], nbf[e, f]
            val = u[e] @ phi[f].T
            dn = torch.einsum("cnk,qka,ca->cnq", u[e], dphi[f], own_n)
            jump, avg = 2 * val, dn.clone()
            for g in range(4):
                at = torch.nonzero((other >= 0) & (of == g)).reshape(-1)
                if not len(at):
                    continue
                un = u[other[at]]
                nn = torch.einsum("cad,cd->ca", jinv[other[at]], n[at])
                jump[at] = val[at] - un @ phi[g].T
                avg[at] = 0.5 * (dn[at] + torch.einsum("cnk,qka,ca->cnq", un, dphi[g], nn))
            own = other < 0
            mate = torch.where(own, torch.arange(e.start, e.stop, device="cuda"), other)
            if helmholtz:
                mate_h = torch.where(own, inv_h[e, f], inv_h[mate, of.clamp(min=0)])
                sigma = factor * 0.5 * (inv_h[e, f] + mate_h)
            else:
                sigma = factor * torch.maximum(tau[e], tau[mate])
            wa = w[None, None, :] * area[f][e][:, None, None]
            y[e] += ((sigma[:, None, None] * jump - avg) * wa) @ phi[f]
            y[e] += torch.einsum("cnq,qka,ca->cnk", -0.5 * jump * wa, dphi[f], own_n)
    return y.reshape(-1)


def _exact_gradient(mlp, X, Y):
    w = torch.from_numpy(mlp.weights()).cuda().bfloat16().double().requires_grad_()
    at, parts = 0, []
    for rows, cols in ((64, 29), (64, 64), (20, 64)):
        m = w[at:at + rows * cols].reshape(rows, cols)
        at += rows * cols
        parts.append((m, w[at:at + rows]))
        at += rows
    h = X.double()
    for k, (m, b) in enumerate(parts):
        h = h @ m.T + b
        if k < 2:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    loss = (h - Y.double()).square().sum(1).mean()
    (g,) = torch.autograd.grad(loss, w)
    return g, float(loss)


def exact(case, seed):
    call = case["call"]
    if call == "solve":
        return None  # an iteration's result, within its tolerance of the solution
    s = prepare(case, seed)
    if call == "vmult":
        m = _mesh(case["mesh"], case["nx"], case["ny"], case["nz"])
        if case["kind"] == "cg":
            return _exact_cg(m, case["degree"], case["components"], s["src"])
        return _exact_dg(m, case["degree"], case["components"], case["kind"] == "helmholtz", s["src"])
    if call == "batch":
        return [_exact_dg(o.mesh, case["degree"], 3, True, x) for o, x in zip(s["batch"].ops, s["src"])]
    return _exact_gradient(s["mlp"], s["X"], s["Y"])


# ---- work --------------------------------------------------------------------------------------


def _operator_work(kind, p, components, nx, ny, nz, size):
    """Vectors once, the mesh (vertices, connectivity) once; multiply-adds of
    the sparse reference gradients, the metric and the P_{p-1} masses."""
    cells = 6 * nx * ny * nz
    vertices = (nx + 1) * (ny + 1) * (nz + 1)
    K = (p + 1) * (p + 2) * (p + 3) // 6
    kq = p * (p + 1) * (p + 2) // 6
    nodes = (p * nx + 1) * (p * ny + 1) * (p * nz + 1) if kind == "cg" else K * cells
    nonzeros = {1: 6, 2: 42, 3: 216}[p]
    flops = 2 * (2 * nonzeros + 9 * kq + 3 * kq * kq)
    if kind != "cg":
        nf, nq = (p + 1) * (p + 2) // 2, p * (p + 1) // 2
        flops += 2 * 4 * (9 * nq + 2 * nf + nf * nf + 2 * nf * nq)
        flops += 2 * K * K if kind == "helmholtz" else 0
    return {"bytes": 2 * size * components * nodes + 3 * size * vertices + 16 * cells + (16 * cells if kind != "cg" else 0),
            "flops": components * cells * flops}


def work(case):
    call = case["call"]
    if call == "vmult":
        return _operator_work(case["kind"], case["degree"], case["components"], case["nx"], case["ny"], case["nz"],
                              8 if case["precision"] == "fp64" else 4)
    if call == "batch":
        each = [_operator_work("helmholtz", case["degree"], 3, n, n, n, 8 if case["precision"] == "fp64" else 4)
                for n in _batch_sizes(case["problems"])]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if call == "solve":
        # about 8 iterations: one FP64 product, and a V-cycle with degree-3 smoothing
        # (6 products on the finest level, as much again on the others)
        n, size = case["n"], 4 if case["levels"] == "fp32" else 8
        outer = _operator_work(case["kind"], case["degree"], 1, n, n, n, 8)
        inner = _operator_work(case["kind"], case["degree"], 1, n, n, n, size)
        return {k: 8 * (outer[k] + 12 * inner[k]) for k in ("bytes", "flops")}
    n = case["samples"]
    return {"bytes": 4 * n * 49 + 4 * 2 * 7380, "flops": 3 * 2 * n * (29 * 64 + 64 * 64 + 64 * 20)}
