#!/usr/bin/env python3
"""Generate the reference-element tables of the tetrahedral Lagrange spaces P1-P3.

Everything is computed in exact rational arithmetic (``fractions.Fraction``)
and only rounded to double when written out.  Two files are produced next to
this script:

* ``ref_tables.h``   constexpr host/device tables (node lattice, nodal-gradient
  matrices, reference masses, face node lists, face masses, p-embeddings);
* ``ref_kernels.cuh`` straight-line device functions that apply those matrices
  with every structural zero removed, every +-1 folded and the terms that
  several rows share formed once (``shared_terms``), so that the cell and face
  kernels run on compile-time constants only.

Conventions (the DoF format every other part of the library relies on)
-----------------------------------------------------------------------
Reference tetrahedron V0=(0,0,0), V1=(1,0,0), V2=(0,1,0), V3=(0,0,1); the
barycentric coordinates are l0 = 1-x-y-z, l1 = x, l2 = y, l3 = z.  A node of
P_q is a multi-index (a0,a1,a2,a3) with sum q and position (a1,a2,a3)/q.
Node order inside a cell: the 4 vertices; then the edges (0,1),(0,2),(0,3),
(1,2),(1,3),(2,3), each walked from its lower to its higher local vertex; then
the faces f=0..3 (face f is opposite vertex f), interior face nodes in
canonical face order; then interior nodes (none for q<=3).  This is the same
vertex/edge/face/interior grouping as deal.II's FE_SimplexP
(FE_SimplexP::FE_SimplexP in deal.II, used at CG/cells_batched/application.cc:1610),
with an edge order of our own.

Canonical face order: the three local vertices of face f in ascending order
(u0<u1<u2); a face node has face-barycentric index b=(a_u0,a_u1,a_u2) and
nodes are sorted by descending b0, then descending b1.  Cells store their
vertices sorted by global vertex id, so both cells that share a face list its
nodes in the same physical order.

P0 (the gradient space of P1) has a single node, the constant function.

Face matrices are normalised so that the integral over a physical face F of a
product of traces equals 2|F| * (the reference-triangle integral), i.e. the
tables already contain the factor 2 and kernels multiply by |F|.
"""
from fractions import Fraction as Fr
from itertools import combinations, product
import math
import os
import random
import sys

# axis order of the six Kuhn tets of a hex (build_kuhn_mesh)
KUHN = [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]
EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]


def face_vertices(f):
    return [v for v in range(4) if v != f]


def nodes(q):
    """Multi-indices (a0,a1,a2,a3) of the P_q Lagrange nodes in cell order."""
    if q == 0:
        return [None]
    out = []
    for i in range(4):
        a = [0, 0, 0, 0]
        a[i] = q
        out.append(tuple(a))
    for (i, j) in EDGES:
        for m in range(1, q):
            a = [0, 0, 0, 0]
            a[i] = q - m
            a[j] = m
            out.append(tuple(a))
    for f in range(4):
        fv = face_vertices(f)
        interior = []
        for a in all_multi(q):
            if a[f] == 0 and all(a[v] >= 1 for v in fv):
                interior.append(a)
        interior.sort(key=lambda a: (-a[fv[0]], -a[fv[1]]))
        out.extend(interior)
    for a in all_multi(q):
        if all(x >= 1 for x in a):
            out.append(a)
    assert len(out) == len(set(out)) == n_nodes(q), (q, len(out))
    return out


def all_multi(q):
    res = []
    for a1 in range(q + 1):
        for a2 in range(q + 1 - a1):
            for a3 in range(q + 1 - a1 - a2):
                res.append((q - a1 - a2 - a3, a1, a2, a3))
    return res


def n_nodes(q):
    return (q + 1) * (q + 2) * (q + 3) // 6


def node_pos(a, q):
    if q == 0:
        return (Fr(1, 4), Fr(1, 4), Fr(1, 4))
    return (Fr(a[1], q), Fr(a[2], q), Fr(a[3], q))


def monomials3(q):
    return [(i, j, k) for i in range(q + 1) for j in range(q + 1 - i)
            for k in range(q + 1 - i - j)]


def monomials2(q):
    return [(i, j) for i in range(q + 1) for j in range(q + 1 - i)]


def solve_inverse(V):
    """Exact inverse of a square Fraction matrix by Gauss-Jordan."""
    n = len(V)
    A = [list(row) + [Fr(int(i == j)) for j in range(n)] for i, row in enumerate(V)]
    for c in range(n):
        p = next(r for r in range(c, n) if A[r][c] != 0)
        A[c], A[p] = A[p], A[c]
        piv = A[c][c]
        A[c] = [x / piv for x in A[c]]
        for r in range(n):
            if r != c and A[r][c] != 0:
                fac = A[r][c]
                A[r] = [x - fac * y for x, y in zip(A[r], A[c])]
    return [row[n:] for row in A]


class Basis3:
    """Lagrange basis of P_q on the reference tet as monomial coefficients."""

    def __init__(self, q):
        self.q = q
        self.nodes = nodes(q)
        self.mono = monomials3(q)
        V = [[mono_eval3(m, node_pos(a, q)) for m in self.mono] for a in self.nodes]
        Vi = solve_inverse(V)
        # phi_n = sum_m Vi[m][n] * mono_m
        self.coef = [[Vi[m][n] for m in range(len(self.mono))] for n in range(len(self.nodes))]

    def value(self, n, x):
        return sum(c * mono_eval3(m, x) for c, m in zip(self.coef[n], self.mono))

    def grad(self, n, a, x):
        s = Fr(0)
        for c, m in zip(self.coef[n], self.mono):
            if m[a] == 0 or c == 0:
                continue
            mm = list(m)
            e = mm[a]
            mm[a] -= 1
            s += c * e * mono_eval3(tuple(mm), x)
        return s

    def poly(self, n):
        return {m: c for c, m in zip(self.coef[n], self.mono) if c != 0}


def mono_eval3(m, x):
    return x[0] ** m[0] * x[1] ** m[1] * x[2] ** m[2]


def tet_int(m):
    """Exact integral of x^i y^j z^k over the reference tet."""
    i, j, k = m
    return Fr(math.factorial(i) * math.factorial(j) * math.factorial(k),
              math.factorial(i + j + k + 3))


def tri_int(m):
    i, j = m
    return Fr(math.factorial(i) * math.factorial(j), math.factorial(i + j + 2))


def poly_mul(p1, p2):
    out = {}
    for m1, c1 in p1.items():
        for m2, c2 in p2.items():
            m = tuple(a + b for a, b in zip(m1, m2))
            out[m] = out.get(m, Fr(0)) + c1 * c2
    return out


def mass3(B1, B2):
    M = []
    for i in range(len(B1.nodes)):
        row = []
        for j in range(len(B2.nodes)):
            pp = poly_mul(B1.poly(i), B2.poly(j))
            row.append(sum(c * tet_int(m) for m, c in pp.items()))
        M.append(row)
    return M


def face_nodes(q, f):
    """Indices (into the cell node list of P_q) of the nodes on face f, canonical order."""
    if q == 0:
        return [0]
    fv = face_vertices(f)
    nl = nodes(q)
    idx = [n for n, a in enumerate(nl) if a[f] == 0]
    idx.sort(key=lambda n: (-nl[n][fv[0]], -nl[n][fv[1]]))
    return idx


class Basis2:
    """Lagrange basis of P_q on the reference triangle in canonical face order."""

    def __init__(self, q):
        self.q = q
        if q == 0:
            self.pts = [(Fr(1, 3), Fr(1, 3))]
            self.coef = [[Fr(1)]]
            self.mono = [(0, 0)]
            self.lattice = [(0, 0, 0)]
            return
        bs = []
        for b0 in range(q, -1, -1):
            for b1 in range(q - b0, -1, -1):
                bs.append((b0, b1, q - b0 - b1))
        self.lattice = bs
        self.pts = [(Fr(b[1], q), Fr(b[2], q)) for b in bs]
        self.mono = monomials2(q)
        V = [[p[0] ** m[0] * p[1] ** m[1] for m in self.mono] for p in self.pts]
        Vi = solve_inverse(V)
        self.coef = [[Vi[m][n] for m in range(len(self.mono))] for n in range(len(self.pts))]

    def poly(self, n):
        return {m: c for c, m in zip(self.coef[n], self.mono) if c != 0}


def mass2(B1, B2):
    M = []
    for i in range(len(B1.coef)):
        row = []
        for j in range(len(B2.coef)):
            pp = poly_mul(B1.poly(i), B2.poly(j))
            row.append(2 * sum(c * tri_int(m) for m, c in pp.items()))
        M.append(row)
    return M


def check_face_trace(q, f):
    """The trace of the 3D basis on face f equals the 2D basis (canonical order)."""
    if q == 0:
        return
    B3 = Basis3(q)
    B2 = Basis2(q)
    fv = face_vertices(f)
    verts = [(Fr(0), Fr(0), Fr(0)), (Fr(1), Fr(0), Fr(0)), (Fr(0), Fr(1), Fr(0)), (Fr(0), Fr(0), Fr(1))]
    fn = face_nodes(q, f)
    # sample points on the face
    for (s, t) in [(Fr(1, 7), Fr(2, 9)), (Fr(3, 11), Fr(1, 5)), (Fr(0), Fr(1, 3))]:
        x = tuple(verts[fv[0]][d] * (1 - s - t) + verts[fv[1]][d] * s + verts[fv[2]][d] * t
                  for d in range(3))
        for i, n in enumerate(fn):
            v3 = B3.value(n, x)
            v2 = sum(c * s ** m[0] * t ** m[1] for c, m in zip(B2.coef[i], B2.mono))
            assert v3 == v2, (q, f, i)
        on = set(fn)
        for n in range(len(B3.nodes)):
            if n not in on:
                assert B3.value(n, x) == 0


def fmt(x):
    v = float(x)
    if v == 0:
        return "0.0"
    return repr(v)


def build(pmax=3):
    data = {}
    for p in range(1, pmax + 1):
        Bp = Basis3(p)
        Bq = Basis3(p - 1) if p > 1 else None
        qnodes = nodes(p - 1) if p > 1 else [None]
        qpos = [node_pos(a, p - 1) if p > 1 else node_pos(None, 0) for a in qnodes]
        K, KQ = n_nodes(p), (n_nodes(p - 1) if p > 1 else 1)
        D = [[[Bp.grad(i, a, qpos[m]) for i in range(K)] for m in range(KQ)] for a in range(3)]
        if p > 1:
            MQ = mass3(Bq, Bq)
        else:
            MQ = [[Fr(1, 6)]]
        MP = mass3(Bp, Bp)
        NF, NFQ = (p + 1) * (p + 2) // 2, (p * (p + 1) // 2 if p > 1 else 1)
        FN = [face_nodes(p, f) for f in range(4)]
        FNQ = [face_nodes(p - 1, f) if p > 1 else [0] for f in range(4)]
        for f in range(4):
            check_face_trace(p, f)
            if p > 1:
                check_face_trace(p - 1, f)
        B2p, B2q = Basis2(p), Basis2(p - 1)
        MFPP = mass2(B2p, B2p)
        MFPQ = mass2(B2p, B2q)
        EMB = None
        if p > 1:
            EMB = [[Bq.value(j, node_pos(Bp.nodes[i], p)) for j in range(KQ)] for i in range(K)]
        # P_{p-1} face basis at the P_p face nodes: MFPQ = MFPP EMBF
        EMBF = [[sum(c * pt[0] ** m[0] * pt[1] ** m[1] for c, m in zip(B2q.coef[j], B2q.mono)) for j in range(NFQ)]
                for pt in B2p.pts]
        for i in range(NF):
            for j in range(NFQ):
                assert MFPQ[i][j] == sum(MFPP[i][k] * EMBF[k][j] for k in range(NF))
        # consistency: D applied to the nodal interpolant of x_a gives 1 for d/dx_a
        for a in range(3):
            lin = [node_pos(nd, p)[a] for nd in Bp.nodes]
            for b in range(3):
                for m in range(KQ):
                    v = sum(D[b][m][i] * lin[i] for i in range(K))
                    assert v == (1 if a == b else 0)
        data[p] = dict(K=K, KQ=KQ, NF=NF, NFQ=NFQ, D=D, MQ=MQ, MP=MP, FN=FN, FNQ=FNQ,
                       MFPP=MFPP, MFPQ=MFPQ, EMB=EMB, EMBF=EMBF, FLAT=B2p.lattice, FLATQ=B2q.lattice,
                       NODES=[node_pos(a, p) for a in Bp.nodes],
                       LATTICE=Bp.nodes, MONO=Bp.mono, COEF=Bp.coef)
    return data


def arr(name, ctype, values, shape):
    def rec(v, depth):
        if depth == len(shape):
            return fmt(v) if ctype == "double" else str(v)
        return "{" + ", ".join(rec(x, depth + 1) for x in v) + "}"
    dims = "".join(f"[{s}]" for s in shape)
    return f"  static constexpr {ctype} {name}{dims} = {rec(values, 0)};\n"


def write_tables(data, path):
    out = []
    out.append("// Generated by gen_tables.py from exact rational arithmetic. Do not edit.\n")
    out.append("// Reference-element tables of the tetrahedral Lagrange spaces P1-P3; the\n")
    out.append("// node, edge and face conventions are documented in gen_tables.py.\n")
    out.append("#pragma once\n\nnamespace sfem {\nnamespace ref {\n\n")
    out.append("template <int P> struct Tables;\n\n")
    for p, d in data.items():
        out.append(f"template <> struct Tables<{p}> {{\n")
        out.append(f"  static constexpr int K = {d['K']};    // P{p} nodes per cell\n")
        out.append(f"  static constexpr int KQ = {d['KQ']};   // P{p-1} nodes (gradient space)\n")
        out.append(f"  static constexpr int NF = {d['NF']};   // P{p} nodes per face\n")
        out.append(f"  static constexpr int NFQ = {d['NFQ']};  // P{p-1} nodes per face\n")
        out.append(arr("NODES", "double", d["NODES"], [d["K"], 3]))
        out.append(arr("LATTICE", "int", [list(a) for a in d["LATTICE"]], [d["K"], 4]))
        out.append(arr("D", "double", d["D"], [3, d["KQ"], d["K"]]))
        out.append(arr("MQ", "double", d["MQ"], [d["KQ"], d["KQ"]]))
        out.append(arr("MP", "double", d["MP"], [d["K"], d["K"]]))
        out.append(arr("FN", "int", d["FN"], [4, d["NF"]]))
        out.append(arr("FNQ", "int", d["FNQ"], [4, d["NFQ"]]))
        out.append(arr("MFPP", "double", d["MFPP"], [d["NF"], d["NF"]]))
        out.append(arr("MFPQ", "double", d["MFPQ"], [d["NF"], d["NFQ"]]))
        if d["EMB"] is not None:
            kq = len(d["EMB"][0])
            out.append(arr("EMB", "double", d["EMB"], [d["K"], kq]))
        # basis polynomials: phi_n(x,y,z) = sum_m COEF[n][m] x^MONO[m][0] y^MONO[m][1] z^MONO[m][2]
        out.append(arr("MONO", "int", [list(m) for m in d["MONO"]], [len(d["MONO"]), 3]))
        out.append(arr("COEF", "double", d["COEF"], [d["K"], len(d["MONO"])]))
        out.append("};\n\n")
    out.append("}  // namespace ref\n}  // namespace sfem\n")
    with open(path, "w") as fh:
        fh.write("".join(out))


def emit_matvec(lines, A, rows, cols, out_expr, in_expr, accumulate, transpose=False):
    """Emit out[r] (+)= sum_c A[r][c] in[c] with zeros removed."""
    nnz = 0
    for r in range(rows):
        terms = []
        for c in range(cols):
            a = A[c][r] if transpose else A[r][c]
            if a == 0:
                continue
            nnz += 1
            x = in_expr(c)
            if a == 1:
                terms.append(("+", x))
            elif a == -1:
                terms.append(("-", x))
            else:
                terms.append(("+", f"T({fmt(a)}) * {x}"))
        o = out_expr(r)
        if not terms:
            if not accumulate:
                lines.append(f"  {o} = T(0);")
            continue
        if accumulate:
            for s, t in terms:
                lines.append(f"  {o} {s}= {t};")
        else:
            s0, t0 = terms[0]
            expr = (t0 if s0 == "+" else f"-({t0})")
            for s, t in terms[1:]:
                expr += f" {s} {t}"
            lines.append(f"  {o} = {expr};")
    return nnz


# ---- products with shared terms ---------------------------------------------------------------
# A product y = A x of a fixed matrix is a straight-line program of multiply-adds.
# Written row by row it costs one operation per non-zero.  Two rows that hold
# the same two inputs in the same ratio can share that pair: t = x_i + r x_j is
# one operation and saves one in every row that uses it.  Pairs are taken
# greedily (most rows first, ties broken at random, the best of many orders
# kept).  For the mass matrices, whose rows are a near-constant background plus
# a few entries, the sums over symmetry classes of nodes (vertices, edges,
# faces) are offered as extra inputs; face masses also in the even and odd
# parts under the reflection that swaps two vertices, which decouple.
# Operations per product (P1 / P2 / P3), row by row -> shared: gradient
# 6/42/216 -> 3/24/113, its transpose 6/42/216 -> 6/36/145, gradient mass
# 1/16/100 -> 1/11/55, cell mass 16/100/400 -> 10/55/153, face mass
# 9/24/88 -> 7/22/66, face value-gradient mass 3/18/60 -> 3/14/43.
# The generators print the counts.


def row_cost(row):
    return max(0, len(row) - (1 if any(abs(c) == 1 for c in row.values()) else 0))


def share_pairs(rows, n_vars, rng):
    """Greedy pair sharing; returns (definitions of the new variables, rows)."""
    rows = [dict(r) for r in rows]
    defs = []
    while True:
        found = {}
        for k, r in enumerate(rows):
            for a, b in combinations(sorted(r), 2):
                found.setdefault((a, b, r[b] / r[a]), []).append(k)
        most = max((len(v) for v in found.values()), default=0)
        if most < 2:
            return defs, rows
        a, b, ratio = key = rng.choice([k for k, v in found.items() if len(v) == most])
        for k in found[key]:
            c = rows[k].pop(a)
            rows[k].pop(b)
            rows[k][n_vars + len(defs)] = c
        defs.append({a: Fr(1), b: ratio})


def sparse_rows(A):
    return [{j: a for j, a in enumerate(r) if a != 0} for r in A]


def with_class_sums(A, classes):
    """Rows over the inputs and one extra input per class: the class's sum."""
    n = len(A[0])
    rows = []
    for r in sparse_rows(A):
        for k, cl in enumerate(classes):
            vals = [r.get(j, Fr(0)) for j in cl]
            c = max(sorted(set(vals)), key=vals.count)
            if c == 0 or vals.count(c) < 2:
                continue
            for j in cl:
                v = r.pop(j, Fr(0)) - c
                if v != 0:
                    r[j] = v
            r[n + k] = c
        rows.append(r)
    return [{j: Fr(1) for j in cl} for cl in classes], rows


def even_odd(A, perm_in, perm_out):
    """Rows for the even and odd parts under a reflection A[po(i)][pi(j)] =
    A[i][j]: extra inputs x_j +- x_pi(j), and for every pair of outputs its even
    and odd half, recombined as (even + odd, even - odd)."""
    n = len(A[0])
    pairs = [(i, perm_in[i]) for i in range(n) if perm_in[i] > i]
    fixed = [i for i in range(n) if perm_in[i] == i]
    extra = [{i: Fr(1), j: Fr(s)} for i, j in pairs for s in (1, -1)]
    rows, place = [], []
    for r in range(len(A)):
        q = perm_out[r]
        if q < r:
            continue
        even = {i: A[r][i] for i in fixed if A[r][i] != 0}
        odd = {}
        for k, (i, j) in enumerate(pairs):
            if A[r][i] + A[r][j] != 0:
                even[n + 2 * k] = (A[r][i] + A[r][j]) / 2
            if A[r][i] != A[r][j]:
                odd[n + 2 * k + 1] = (A[r][i] - A[r][j]) / 2
        rows.append(even)
        if q == r:
            place.append((r, len(rows) - 1, None))
        else:
            rows.append(odd)
            place.append((r, len(rows) - 2, 1))
            place.append((q, len(rows) - 2, -1))
    return extra, rows, place


def shared_terms(A, classes=(), reflections=(), tries=60, seed=0):
    """The cheapest program found for y = A x: (cost, definitions, rows), variables
    numbered inputs first, then definitions in order."""
    n = len(A[0])
    forms = [([], sparse_rows(A), None)]
    for k in range(1, len(classes) + 1):
        forms += [(*with_class_sums(A, sub), None) for sub in combinations(classes, k)]
    forms += [even_odd(A, pi, po) for pi, po in reflections]
    rng = random.Random(seed)
    best = None
    for extra, rows, place in forms:
        for _ in range(tries):
            defs, out = share_pairs(rows, n + len(extra), rng)
            defs = extra + defs
            if place is not None:
                defs = defs + out
                base = n + len(defs) - len(out)
                at = [None] * len(A)
                for r, k, sign in place:
                    at[r] = {base + k: Fr(1)} if sign is None else {base + k: Fr(1), base + k + 1: Fr(sign)}
                out = at
            cost = sum(map(row_cost, defs)) + sum(map(row_cost, out))
            if best is None or cost < best[0]:
                best = (cost, defs, out)
    check_program(A, best[1], best[2])
    return best


def check_program(A, defs, rows):
    """The program is A, exactly."""
    n = len(A[0])
    val = [[Fr(int(i == j)) for j in range(n)] for i in range(n)]

    def lin(r):
        return [sum((c * val[v][j] for v, c in r.items()), Fr(0)) for j in range(n)]

    for d in defs:
        val.append(lin(d))
    for r, want in zip(rows, A):
        assert lin(r) == list(want)


def emit_program(lines, program, n, out_expr, in_expr, accumulate):
    """Emit the program; every definition right before its first use."""
    _, defs, rows = program
    done = set()

    def name(v):
        return in_expr(v) if v < n else f"t{v - n}"

    def expr(r):
        terms = sorted(r.items(), key=lambda vc: (abs(vc[1]) != 1, vc[1] < 0, vc[0]))
        out = []
        for v, c in terms:
            if abs(c) == 1:
                out.append(("+" if c > 0 else "-", name(v)))
            else:
                out.append(("+", f"T({fmt(c)}) * {name(v)}"))
        return out

    def join(terms):
        s = terms[0][1] if terms[0][0] == "+" else f"-({terms[0][1]})"
        return s + "".join(f" {sg} {t}" for sg, t in terms[1:])

    def need(r):
        for v in sorted(r):
            if v >= n and v not in done:
                done.add(v)
                need(defs[v - n])
                lines.append(f"  const T t{v - n} = {join(expr(defs[v - n]))};")

    for k, r in enumerate(rows):
        need(r)
        if not r:
            if not accumulate:
                lines.append(f"  {out_expr(k)} = T(0);")
        elif accumulate:
            for sg, t in expr(r):
                lines.append(f"  {out_expr(k)} {sg}= {t};")
        else:
            lines.append(f"  {out_expr(k)} = {join(expr(r))};")


def node_classes(lattice, q):
    """Nodes by kind (vertex, edge, face), kinds of at least two nodes."""
    kinds = {}
    for i, a in enumerate(lattice):
        kinds.setdefault(sum(1 for x in a if x > 0), []).append(i)
    return [v for _, v in sorted(kinds.items()) if len(v) > 1 and q > 0]


def swap_perm(lattice, i, j):
    def sw(a):
        a = list(a)
        a[i], a[j] = a[j], a[i]
        return tuple(a)
    return [lattice.index(sw(a)) for a in map(tuple, lattice)]


def write_kernels(data, path):
    L = []
    L.append("// Generated by gen_tables.py from exact rational arithmetic. Do not edit.")
    L.append("// Straight-line applications of the reference matrices of ref_tables.h:")
    L.append("// structural zeros are removed, +-1 entries folded and terms that several rows")
    L.append("// share formed once (t..), so cell and face kernels issue only additions and FMAs")
    L.append("// on compile-time constants, about 0.6 of the operations of the plain rows for P3.")
    L.append("#pragma once\n")
    L.append("namespace sfem {\nnamespace gen {\n")
    stats = []
    for p, d in data.items():
        K, KQ, NF, NFQ = d["K"], d["KQ"], d["NF"], d["NFQ"]
        kq = p - 1
        lat, latq = list(d["LATTICE"]), (nodes(kq) if kq > 0 else [(0, 0, 0, 0)])
        refl = (swap_perm(d["FLAT"], 0, 1), swap_perm(d["FLATQ"], 0, 1))

        def fn(doc, sig, body):
            L.append(f"// P{p}: {doc}")
            L.append(f"template <typename T{', typename F' if 'F&&' in sig else ''}> __host__ __device__ __forceinline__ void {sig} {{")
            L.extend(body)
            L.append("}")

        def product_fn(doc, sig, A, out_expr, in_expr, accumulate=False, classes=(), reflections=(), post=()):
            prog = shared_terms(A, classes, reflections, tries=60 if len(A) < 16 else 30)
            nonzeros = sum(1 for r in A for a in r if a != 0)
            stats.append((p, sig.split("_P")[0], prog[0] + (sum(1 for r in prog[2] if any(abs(c) == 1 for c in r.values())) if accumulate else 0), nonzeros))
            body = []
            emit_program(body, prog, len(A[0]), out_expr, in_expr, accumulate)
            fn(doc, sig, body + list(post))

        # nodal gradient: g[a][m] = sum_i D[a][m][i] u[i]
        DD = [row for a in range(3) for row in d["D"][a]]
        product_fn(f"reference gradient in the P{p-1} nodal basis, g[a*{KQ}+m] = (D_a u)_m",
                   f"grad_P{p}(const T (&u)[{K}], T (&g)[{3*KQ}])", DD, lambda r: f"g[{r}]", lambda c: f"u[{c}]")
        # y[i] += sum_{a,m} D[a][m][i] h[a*KQ+m]
        product_fn("y += sum_a D_a^T h_a", f"gradT_P{p}(const T (&h)[{3*KQ}], T (&y)[{K}])",
                   [list(c) for c in zip(*DD)], lambda r: f"y[{r}]", lambda c: f"h[{c}]", accumulate=True)
        product_fn(f"o = MQ w (reference-tet mass of P{p-1}), one gradient component",
                   f"massQ_P{p}(const T* w, T* o)", d["MQ"], lambda r: f"o[{r}]", lambda c: f"w[{c}]",
                   classes=node_classes(latq, kq))
        prog = shared_terms([list(c) for c in zip(*DD)], tries=60 if K < 16 else 30)
        body = []
        emit_program(body, prog, 3 * KQ, lambda r: f"y({r})", lambda c: f"h[{c}]", True)
        fn("y(i) += (sum_a D_a^T h_a)_i", f"gradTInto_P{p}(const T (&h)[{3*KQ}], F&& y)", body)
        # seen from a face: nodes by layers from the face (layer l: l nodes' worth of
        # the opposite vertex), each layer in canonical face order, vertices (v0, v1,
        # v2, opposite); the same formulas then hold for all four faces
        lat_side = sorted(lat, key=lambda a: (a[3], -a[0], -a[1]))
        d["SIDE"] = []
        for f in range(4):
            v = [x for x in range(4) if x != f] + [f]
            rows = []
            for a in lat_side:
                b = [0, 0, 0, 0]
                for k in range(4):
                    b[v[k]] = a[k]
                rows.append(lat.index(tuple(b)))
            assert rows[:NF] == d["FN"][f]
            d["SIDE"].append(rows)
        # derivatives along v_w - opposite vertex at the P_{p-1} face nodes (face 3), for
        # the one-launch DG P3 form
        if p == 3:
            side = d["SIDE"][3]
            along = []
            for w in range(3):
                for m in d["FNQ"][3]:
                    row = [(d["D"][w - 1][m][i] if w else Fr(0)) - d["D"][2][m][i] for i in range(K)]
                    along.append([row[side[i]] for i in range(K)])
            product_fn(f"g[w*{NFQ}+m] = derivative along v_w - o at face node m, from a cell's values in side order",
                       f"sideGrad_P{p}(const T* s, T* g)", along, lambda r: f"g[{r}]", lambda c: f"s[{c}]")
        # the same three row by row, for the CG kernels that run out of registers
        # before they run out of arithmetic (see cg_local_apply)
        body = []
        for a in range(3):
            emit_matvec(body, d["D"][a], KQ, K, lambda r, a=a: f"g[{a*KQ + r}]", lambda c: f"u[{c}]", False)
        fn("grad, row by row", f"gradRows_P{p}(const T (&u)[{K}], T (&g)[{3*KQ}])", body)
        body = []
        emit_matvec(body, [list(c) for c in zip(*DD)], K, 3 * KQ, lambda r: f"y[{r}]", lambda c: f"h[{c}]", True)
        fn("gradT, row by row", f"gradTRows_P{p}(const T (&h)[{3*KQ}], T (&y)[{K}])", body)
        body = []
        emit_matvec(body, d["MQ"], KQ, KQ, lambda r: f"o[{r}]", lambda c: f"w[{c}]", False)
        fn("massQ, row by row", f"massQRows_P{p}(const T* w, T* o)", body)
        # y += s * MP u: t = MP u, then scaled
        prog = shared_terms(d["MP"], node_classes(lat, p), [(swap_perm(lat, 0, 1),) * 2] if p > 1 else (), tries=10)
        stats.append((p, "massP", prog[0], K * K))
        body = [f"  T o[{K}];"]
        emit_program(body, prog, K, lambda r: f"o[{r}]", lambda c: f"u[{c}]", False)
        body.append(f"  for (int i = 0; i < {K}; ++i) y[i] += s * o[i];")
        fn(f"y += s MP u (reference-tet mass of P{p})", f"massP_P{p}(const T* u, T s, T* y)", body)
        fcl = node_classes(d["FLAT"], p)
        product_fn(f"o = MFPP j (face mass P{p} x P{p}, factor 2 included)", f"facePP_P{p}(const T* j, T* o)", d["MFPP"],
                   lambda r: f"o[{r}]", lambda c: f"j[{c}]", classes=fcl, reflections=[(refl[0], refl[0])])
        fqcl = node_classes(d["FLATQ"], p - 1)
        product_fn(f"o += MFPQ a (face mass P{p} x P{p-1})", f"facePQ_P{p}(const T* a, T* o)", d["MFPQ"],
                   lambda r: f"o[{r}]", lambda c: f"a[{c}]", accumulate=True, classes=fqcl)
        product_fn(f"o = MFPQ^T j (face mass P{p-1} x P{p})", f"faceQP_P{p}(const T* j, T* o)",
                   [list(c) for c in zip(*d["MFPQ"])], lambda r: f"o[{r}]", lambda c: f"j[{c}]", classes=fcl)
        # the face terms of the DG apply: the factors 1/4 of the averages and of the
        # gradient test are in the matrices
        quarter = [[-a / 4 for a in r] for r in d["MFPQ"]]
        product_fn("o(i) += (-1/4 MFPQ a)_i", f"faceFlux_P{p}(const T* a, F&& o)", quarter,
                   lambda r: f"o({r})", lambda c: f"a[{c}]", accumulate=True, classes=fqcl)
        product_fn(f"o = -1/4 MFPQ^T j from t = MFPP j (MFPQ = MFPP E, E the P{p-1} face basis at the P{p} nodes)",
                   f"faceTest_P{p}(const T* t, T* o)", [[-a / 4 for a in c] for c in zip(*d["EMBF"])],
                   lambda r: f"o[{r}]", lambda c: f"t[{c}]")
        L.append("")
    # single-row functions for warp-split kernels: a switch on the row index
    # that folds away once the caller's loops are unrolled
    for p, d in data.items():
        K, KQ, NF, NFQ = d["K"], d["KQ"], d["NF"], d["NFQ"]

        def row_switch(name, sig, rows, body_of_row):
            L.append(f"template <typename T> __host__ __device__ __forceinline__ T {name}({sig}) {{")
            L.append("  switch (r) {")
            for r in range(rows):
                L.append(f"    case {r}: return {body_of_row(r)};")
            L.append("  }")
            L.append("  return T(0);")
            L.append("}")

        def lin(coefs, term):
            parts = []
            for c, a in coefs:
                if a == 0:
                    continue
                t = term(c)
                if a == 1:
                    parts.append(f"+ {t}")
                elif a == -1:
                    parts.append(f"- {t}")
                else:
                    parts.append(f"+ T({fmt(a)}) * {t}")
            if not parts:
                return "T(0)"
            s = " ".join(parts)
            return s[2:] if s.startswith("+ ") else "-" + s[2:] if False else ("T(0) " + s if s.startswith("-") else s[2:])

        # grad row r = a*KQ + m from u[i*us]
        row_switch(f"grad_row_P{p}", "int r, const T* u, int us", 3 * KQ,
                   lambda r: lin([(i, d["D"][r // KQ][r % KQ][i]) for i in range(K)], lambda i: f"u[{i} * us]"))
        # gradT row i from h[(a*KQ+m)*hs]
        row_switch(f"gradT_row_P{p}", "int r, const T* h, int hs", K,
                   lambda i: lin([(a * KQ + m, d["D"][a][m][i]) for a in range(3) for m in range(KQ)],
                                 lambda c: f"h[{c} * hs]"))
        # MQ row m from w[n]
        row_switch(f"massQ_row_P{p}", "int r, const T* w", KQ,
                   lambda m: lin([(n, d["MQ"][m][n]) for n in range(KQ)], lambda n: f"w[{n}]"))
        # MP row i from u[j*us]
        row_switch(f"massP_row_P{p}", "int r, const T* u, int us", K,
                   lambda i: lin([(j, d["MP"][i][j]) for j in range(K)], lambda j: f"u[{j} * us]"))
        # position of cell node i on face f (P_p) / of P_{p-1} node m on face f, -1 if absent
        cases = " ".join(f"case {f*K+i}: return {d['FN'][f].index(i) if i in d['FN'][f] else -1};"
                         for f in range(4) for i in range(K))
        L.append(f"__host__ __device__ __forceinline__ constexpr int face_pos_P{p}(int f, int i) "
                 f"{{ switch (f * {K} + i) {{ {cases} }} return -1; }}")
        cases = " ".join(f"case {f*KQ+m}: return {d['FNQ'][f].index(m) if m in d['FNQ'][f] else -1};"
                         for f in range(4) for m in range(KQ))
        L.append(f"__host__ __device__ __forceinline__ constexpr int faceq_pos_P{p}(int f, int m) "
                 f"{{ switch (f * {KQ} + m) {{ {cases} }} return -1; }}")
        L.append("")
    # dispatch struct and runtime face-node tables
    for p, d in data.items():
        K, KQ, NF, NFQ = d["K"], d["KQ"], d["NF"], d["NFQ"]
        L.append(f"// P{p} face node lists for runtime (neighbour) face indices")
        fn = ", ".join("{" + ", ".join(str(x) for x in row) + "}" for row in d["FN"])
        L.append(f"static __constant__ int8_t cFN_P{p}[4][{NF}] = {{{fn}}};")
    L.append("")
    L.append("template <int P> struct Ops;")
    for p, d in data.items():
        K, KQ, NF, NFQ = d["K"], d["KQ"], d["NF"], d["NFQ"]
        L.append(f"template <> struct Ops<{p}> {{")
        L.append(f"  static constexpr int K = {K}, KQ = {KQ}, NF = {NF}, NFQ = {NFQ};")
        L.append(f"  template <class T> static __device__ __forceinline__ void grad(const T (&u)[{K}], T (&g)[{3*KQ}]) {{ grad_P{p}(u, g); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void gradT(const T (&h)[{3*KQ}], T (&y)[{K}]) {{ gradT_P{p}(h, y); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void gradRows(const T (&u)[{K}], T (&g)[{3*KQ}]) {{ gradRows_P{p}(u, g); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void gradTRows(const T (&h)[{3*KQ}], T (&y)[{K}]) {{ gradTRows_P{p}(h, y); }}")
        L.append(f"  template <class T, class F> static __device__ __forceinline__ void gradTInto(const T (&h)[{3*KQ}], F&& y) {{ gradTInto_P{p}(h, y); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void massQRows(const T* w, T* o) {{ massQRows_P{p}(w, o); }}")
        L.append(f"  template <class T, class F> static __device__ __forceinline__ void faceFlux(const T* a, F&& o) {{ faceFlux_P{p}(a, o); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void faceTest(const T* t, T* o) {{ faceTest_P{p}(t, o); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void massQ(const T* w, T* o) {{ massQ_P{p}(w, o); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void massP(const T* u, T s, T* y) {{ massP_P{p}(u, s, y); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void facePP(const T* j, T* o) {{ facePP_P{p}(j, o); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void facePQ(const T* a, T* o) {{ facePQ_P{p}(a, o); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ void faceQP(const T* j, T* o) {{ faceQP_P{p}(j, o); }}")
        L.append(f"  static __device__ __forceinline__ int fn_runtime(int f, int i) {{ return cFN_P{p}[f][i]; }}")
        L.append(f"  template <class T> static __device__ __forceinline__ T grad_row(int r, const T* u, int us) {{ return grad_row_P{p}(r, u, us); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ T gradT_row(int r, const T* h, int hs) {{ return gradT_row_P{p}(r, h, hs); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ T massQ_row(int r, const T* w) {{ return massQ_row_P{p}(r, w); }}")
        L.append(f"  template <class T> static __device__ __forceinline__ T massP_row(int r, const T* u, int us) {{ return massP_row_P{p}(r, u, us); }}")
        L.append(f"  static __host__ __device__ __forceinline__ constexpr int face_pos(int f, int i) {{ return face_pos_P{p}(f, i); }}")
        L.append(f"  static __host__ __device__ __forceinline__ constexpr int faceq_pos(int f, int m) {{ return faceq_pos_P{p}(f, m); }}")
        cases = " ".join(f"case {f*NF+i}: return {d['FN'][f][i]};" for f in range(4) for i in range(NF))
        L.append(f"  static __host__ __device__ __forceinline__ constexpr int fn(int f, int i) {{ switch (f * {NF} + i) {{ {cases} }} return 0; }}")
        if p == 3:
            L.append(f"  template <class T> static __device__ __forceinline__ void sideGrad(const T* s, T* g) {{ sideGrad_P{p}(s, g); }}")
            cases = " ".join(f"case {f*K+i}: return {d['SIDE'][f][i]};" for f in range(4) for i in range(K))
            L.append(f"  static __host__ __device__ __forceinline__ constexpr int side(int f, int i) {{ switch (f * {K} + i) {{ {cases} }} return 0; }}")
        # Kuhn hex: lattice offset (x, y, z in 0..p) of node i of tet q.  Tet q walks
        # the hex edges in axis order KUHN[q], which is also the order of its
        # (ascending) vertices.
        hexn = []
        for q in range(6):
            for a in d["LATTICE"]:
                off = [0, 0, 0]
                for s, axis in enumerate(KUHN[q]):
                    off[axis] = sum(a[s + 1:])
                hexn.append(off[0] + (p + 1) * (off[1] + (p + 1) * off[2]))
        cases = " ".join(f"case {k}: return {v};" for k, v in enumerate(hexn))
        L.append(f"  static __host__ __device__ __forceinline__ constexpr int hex_node(int q, int i) {{ switch (q * {K} + i) {{ {cases} }} return 0; }}")
        cases = " ".join(f"case {f*NFQ+i}: return {d['FNQ'][f][i]};" for f in range(4) for i in range(NFQ))
        L.append(f"  static __host__ __device__ __forceinline__ constexpr int fnq(int f, int m) {{ switch (f * {NFQ} + m) {{ {cases} }} return 0; }}")
        L.append("};")
    L.append("")
    L.append("}  // namespace gen\n}  // namespace sfem")
    with open(path, "w") as fh:
        fh.write("\n".join(L) + "\n")
    return stats


def main():
    here = os.path.dirname(os.path.abspath(__file__))
    data = build()
    write_tables(data, os.path.join(here, "ref_tables.h"))
    stats = write_kernels(data, os.path.join(here, "ref_kernels.cuh"))
    for s in stats:
        print("P%d %-10s %4d operations for %4d non-zeros" % s)


if __name__ == "__main__":
    sys.exit(main())
