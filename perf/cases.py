"""Assembly workloads for timing the engine through its public C ABI binding.

Every case builds a finite-element problem on a seeded jittered mesh (element
groups as the weak-form lowering hands them to the engine: Gauss points,
form-function tables per orientation, coefficient programs, DOF addresses) and
runs one of the calls an application makes with it:

  step      slgpu_matrix_process on a resident pattern, result taken as device
            CSR; with new per-element coefficients uploaded first
            (data = "element") or unchanged inputs (data = "resident"), and
            followed by the device elimination of the constrained DOFs
            (eliminate)
  sweep     the same with new term scales: one frequency of a harmonic problem
  generate  a matrix created, its groups added, processed on the resident
            pattern and its values downloaded: generate() + A() of a
            formulation assembled again and again
  first     the same with DOF numbers no earlier call had, so the pattern is
            built, the CSR structure and values taken on the device: the first
            assembly, or one after the mesh or the fields changed
  rhs       the right-hand side of one field with an interpolated source
  serve     a burst of requests with new coefficients on resident templates

Physics and sizes follow the benchmark's workloads: Poisson on quadrangles
(order 1, 256 x 256), order-2 elasticity on hexahedra, p-adaptive Helmholtz on
tetrahedra of orders 1 to 5, harmonic eddy currents with order-2 edge elements,
and the mixed serving pool.
"""
from __future__ import annotations

import ctypes
import itertools
import math
from ctypes import POINTER, c_int64, c_uint8, c_void_p

import numpy as np
import torch

from sparselizard_b200 import abi, serving

PRECISION = {"fp64": abi.PREC_FP64, "split": abi.PREC_SPLIT, "fp32": abi.PREC_FP32}
QUAD, TET, HEX = 3, 4, 5  # element type numbers of the ABI
BURST_TEMPLATES = 4


# ---------------------------------------------------------------- the cases

def _case(name, call, problem, cell, order, n, precision, **more):
    c = dict(name=name, call=call, problem=problem, cell=cell, order=order, n=n, precision=precision,
             data="resident", eliminate=False, requests=0)
    c.update(more)
    return c


def listed():
    return [
        # Interactive or inner-loop assembly of a small 2D problem whose material changes every step: launches and latency.
        _case("poisson_quad_small", "step", "poisson", "quad", 1, 13, "fp64", data="element"),
        # The benchmark's 2D problem, handed to a device solver: values, then the elimination of the Dirichlet DOFs.
        _case("poisson_quad_256", "step", "poisson", "quad", 1, 256, "fp64", eliminate=True),
        # Higher-order 2D diffusion with new coefficients per step (nonlinear material), in plain FP64.
        _case("diffusion_quad_p3", "step", "poisson", "quad", 3, 149, "fp64", data="element"),
        # The headline problem, order-2 elasticity on hexahedra, in split precision: large, the whole step on the device.
        _case("elasticity_hex_48", "step", "elasticity", "hex", 2, 48, "split"),
        # The same in plain FP64 at an odd size.
        _case("elasticity_hex_27_fp64", "step", "elasticity", "hex", 2, 27, "fp64"),
        # FP32-level tier (float element matrices) on unstructured order-2 tetrahedra.
        _case("elasticity_tet_fp32", "step", "elasticity", "tet", 2, 14, "fp32"),
        # p-adaptive Helmholtz: groups of orders 1 to 5 of very different shapes in one step.
        _case("helmholtz_tet_p1_5", "step", "helmholtz", "tet", 5, 20, "split"),
        # Frequency sweep of harmonic eddy currents with order-2 edge elements: new scales, then the step.
        _case("eddy_tet_sweep", "sweep", "eddy", "tet", 2, 20, "split"),
        # Repeated generate() + A(): lowering uploaded again, values downloaded into the caller's page-locked array.
        _case("generate_hex_16", "generate", "elasticity", "hex", 2, 16, "split"),
        # First assembly, or the first after the numbering changed: the symbolic phase, for a device solver.
        _case("first_hex_15", "first", "elasticity", "hex", 2, 15, "split"),
        # Right-hand side with an interpolated source field.
        _case("rhs_hex_41", "rhs", "poisson", "hex", 2, 41, "fp64"),
        # Serving: a burst of requests with new coefficient fields on resident problems of four kinds.
        _case("serve_burst_16", "serve", "pool", "mixed", 2, 10, "split", requests=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges: sizes log-uniform per call, problem and order."""
    call = rng.choice(["step", "step", "step", "step", "sweep", "generate", "first", "rhs", "serve"])
    precision = rng.choice(["fp64", "split", "split", "fp32"])
    if call == "serve":
        c = _case("", call, "pool", "mixed", 2, _log_int(rng, 4, 14), rng.choice(["fp64", "split"]), requests=rng.randint(3, 24))
    elif call == "sweep":
        c = _case("", call, "eddy", "tet", rng.choice([1, 2]), _log_int(rng, 3, 20), precision)
    elif call == "rhs":
        cell, order = rng.choice([("quad", 1), ("quad", 2), ("quad", 3), ("hex", 1), ("hex", 2)])
        c = _case("", call, "poisson", cell, order, _log_int(rng, 5, 45) if cell == "hex" else _log_int(rng, 9, 400), "fp64")
    elif call in ("generate", "first"):
        problem, cell, order, lo, hi = rng.choice([("elasticity", "hex", 2, 4, 18), ("elasticity", "hex", 1, 4, 32),
                                                   ("poisson", "quad", 2, 9, 250), ("poisson", "tet", 2, 4, 20),
                                                   ("helmholtz", "tet", 4, 4, 12)])
        c = _case("", call, problem, cell, order, _log_int(rng, lo, hi), precision)
    else:
        problem, cell, order, lo, hi = rng.choice([
            ("poisson", "quad", 1, 5, 500), ("poisson", "quad", 2, 5, 350), ("poisson", "quad", 3, 5, 200),
            ("poisson", "hex", 1, 4, 70), ("poisson", "hex", 2, 4, 45), ("poisson", "tet", 3, 3, 20),
            ("elasticity", "hex", 1, 4, 60), ("elasticity", "hex", 2, 4, 44), ("elasticity", "tet", 2, 4, 24),
            ("helmholtz", "tet", 5, 4, 20), ("helmholtz", "tet", 3, 4, 24)])
        c = _case("", call, problem, cell, order, _log_int(rng, lo, hi), precision,
                  data=rng.choice(["resident", "element"]), eliminate=rng.random() < 0.3)
    del c["name"]
    return c


# ---------------------------------------------------------------- form functions

def _legendre(k, x, scale=1.0):
    """Scaled Legendre polynomial scale^k P_k(x / scale) and its derivatives with respect to x and scale."""
    p, px, ps = [np.ones_like(x), x], [np.zeros_like(x), np.ones_like(x)], [np.zeros_like(x), np.zeros_like(x)]
    s = scale + np.zeros_like(x)
    for m in range(2, k + 1):
        a, b = (2 * m - 1) / m, (m - 1) / m
        p.append(a * x * p[-1] - b * s * s * p[-2])
        px.append(a * (p[m - 1] + x * px[-1]) - b * s * s * px[-2])
        ps.append(a * x * ps[-1] - b * (2 * s * p[m - 2] + s * s * ps[-2]))
    return p[k], px[k], ps[k]


def _line(order, x):
    """Hierarchical functions on [-1, 1]: two vertices, then bubbles of degree 2 .. order; values and derivatives [functions][points]."""
    v, d = [(1 - x) / 2, (1 + x) / 2], [-0.5 + 0 * x, 0.5 + 0 * x]
    for k in range(2, order + 1):
        pk, dk, _ = _legendre(k, x)
        pm, dm, _ = _legendre(k - 2, x)
        v.append((pk - pm) / math.sqrt(2 * (2 * k - 1)))
        d.append((dk - dm) / math.sqrt(2 * (2 * k - 1)))
    return np.array(v), np.array(d)


def _grid_cell(dim, order):
    """Gauss points, weights, geometry tables and H1 tables [1 + dim][functions][points] of the tensor-product cell."""
    x, w = np.polynomial.legendre.leggauss(order + 1)
    pts = np.array(list(itertools.product(x, repeat=dim)))[:, ::-1]
    weights = np.array([np.prod(t) for t in itertools.product(w, repeat=dim)])
    corners = [(0, 0), (1, 0), (1, 1), (0, 1)]
    geo = corners if dim == 2 else [c + (z,) for z in (0, 1) for c in corners]
    fun = [t[::-1] for t in itertools.product(range(order + 1), repeat=dim)]

    def tables(which, p):
        one = [_line(p, pts[:, k]) for k in range(dim)]
        out = []
        for deriv in range(-1, dim):
            out.append([np.prod([one[k][1 if k == deriv else 0][f[k]] for k in range(dim)], axis=0) for f in which])
        return np.array(out)

    return weights, geo, tables(geo, 1), fun, tables(fun, order)


def _tet_points(m):
    """Collapsed Gauss points (barycentric coordinates) and weights on the reference tetrahedron."""
    x, w = np.polynomial.legendre.leggauss(m)
    x, w = (x + 1) / 2, w / 2
    lam, weights = [], []
    for (a, wa), (b, wb), (c, wc) in itertools.product(zip(x, w), repeat=3):
        k, e, p = a, b * (1 - a), c * (1 - a) * (1 - b)
        lam.append((1 - k - e - p, k, e, p))
        weights.append(wa * wb * wc * (1 - a) ** 2 * (1 - b))
    return np.array(lam).T, np.array(weights)


EDGES = list(itertools.combinations(range(4), 2))
FACES = list(itertools.combinations(range(4), 3))


class _Poly:
    """A function of the barycentric coordinates: its values and its derivatives with respect to each of them."""

    def __init__(self, v, d):
        self.v, self.d = v, d

    def __mul__(self, o):
        return _Poly(self.v * o.v, [a * o.v + self.v * b for a, b in zip(self.d, o.d)])


def _kernel(lam, i, j, k):
    """Scaled Legendre polynomial of degree k in lam_j - lam_i."""
    v, dx, ds = _legendre(k, lam[j] - lam[i], lam[i] + lam[j])
    d = [np.zeros_like(v) for _ in range(4)]
    d[j], d[i] = dx + ds, ds - dx
    return _Poly(v, d)


def _tet_h1(lam, order):
    """H1 functions of sorted vertices, in the order vertices, edges, faces, cell: [(entity kind, entity, number, function)]."""
    one = [_Poly(lam[i], [np.ones_like(lam[i]) * (k == i) for k in range(4)]) for i in range(4)]
    out = [("v", i, 0, one[i]) for i in range(4)]
    for e, (i, j) in enumerate(EDGES):
        out += [("e", e, k, one[i] * one[j] * _kernel(lam, i, j, k)) for k in range(order - 1)]
    for f, (i, j, k) in enumerate(FACES):
        powers = [(a, d - a) for d in range(max(0, order - 2)) for a in range(d + 1)]
        out += [("f", f, m, one[i] * one[j] * one[k] * _kernel(lam, i, j, a) * _kernel(lam, i, k, b)) for m, (a, b) in enumerate(powers)]
    powers = [(a, b, d - a - b) for d in range(max(0, order - 3)) for a in range(d + 1) for b in range(d - a + 1)]
    bubble = one[0] * one[1] * one[2] * one[3]
    out += [("c", 0, m, bubble * _kernel(lam, 0, 1, a) * _kernel(lam, 0, 2, b) * _kernel(lam, 0, 3, c)) for m, (a, b, c) in enumerate(powers)]
    return out


# Reference gradients of the barycentric coordinates (1 - k - e - p, k, e, p).
GRAD = np.array([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
PERMS = list(itertools.permutations(range(4)))


def _tet_h1_tables(order, lam, perm):
    """Values and reference derivatives [4][functions][points] for elements whose k-th smallest vertex is local vertex perm[k]."""
    fs = _tet_h1([lam[p] for p in perm], order)
    g = GRAD[list(perm)]
    return np.array([[f[3].v for f in fs]] + [[sum(f[3].d[k] * g[k, a] for k in range(4)) for f in fs] for a in range(3)])


def _tet_curl_tables(order, lam, perm):
    """Edge-element functions and their curls [6][functions][points] (order 1: 6 functions, order 2: 20)."""
    lam, g = [lam[p] for p in perm], GRAD[list(perm)]
    fun, cur = [], []
    for i, j in EDGES:
        fun.append(lam[i] * g[j][:, None] - lam[j] * g[i][:, None])
        cur.append(2 * np.cross(g[i], g[j])[:, None] + 0 * lam[i])
        if order > 1:
            fun.append(lam[i] * g[j][:, None] + lam[j] * g[i][:, None])
            cur.append(np.zeros((3, lam[i].size)))
    if order > 1:
        for i, j, k in FACES:
            for a, b, c in ((i, j, k), (j, i, k)):  # lam_a (lam_b grad lam_c - lam_c grad lam_b)
                fun.append(lam[a] * (lam[b] * g[c][:, None] - lam[c] * g[b][:, None]))
                ga, gb, gc = g[a][:, None], g[b][:, None], g[c][:, None]
                cross = lambda x, y: np.cross(x, y, axis=0)  # noqa: E731
                cur.append(lam[b] * cross(ga, gc) - lam[c] * cross(ga, gb) + 2 * lam[a] * cross(gb, gc))
    return np.concatenate([np.array(fun).transpose(1, 0, 2), np.array(cur).transpose(1, 0, 2)])


# ---------------------------------------------------------------- meshes and DOF numbers

class _Mesh:
    pass


def _grid(dim, n, order, components):
    """Structured quadrangles or hexahedra; H1 numbers by component, then kind of entity, then position."""
    m = _Mesh()
    m.dim, m.type, m.components = dim, (QUAD if dim == 2 else HEX), components
    weights, geo, lagrange, fun, tab = _grid_cell(dim, order)
    cell = np.stack(np.meshgrid(*[np.arange(n)] * dim, indexing="ij")).reshape(dim, -1)[::-1]  # x fastest
    m.nelem = cell.shape[1]
    stride = (n + 1) ** np.arange(dim)
    m.conn = np.stack([((cell + np.array(c)[:, None]) * stride[:, None]).sum(0) for c in geo], axis=1).astype(np.int32)
    nodes = np.stack(np.meshgrid(*[np.arange(n + 1)] * dim, indexing="ij")).reshape(dim, -1)[::-1]
    m.grid, m.h = nodes.T / n, 1.0 / n
    start, total, addr, fixed = {}, 0, [], []
    for kinds in itertools.product(range(order), repeat=dim):  # 0: vertex, k: bubble k, per direction
        size = [n + 1 if k == 0 else n for k in kinds]
        start[kinds] = (total, size)
        pos = np.stack(np.meshgrid(*[np.arange(s) for s in size], indexing="ij")).reshape(dim, -1)
        last = dim - 1
        edge = (pos[last] == 0) & (kinds[last] == 0)
        if components == 1:
            for k in range(dim):
                edge |= (kinds[k] == 0) & ((pos[k] == 0) | (pos[k] == size[k] - 1))
        flat = sum(pos[k] * int(np.prod(size[:k])) for k in range(dim))
        fixed.append(total + flat[edge])
        total += int(np.prod(size))
    for f in fun:
        base, size = start[tuple(max(0, k - 1) for k in f)]
        pos = [cell[k] + (f[k] == 1) for k in range(dim)]
        addr.append(base + sum(pos[k] * int(np.prod(size[:k])) for k in range(dim)))
    addr, fixed = np.array(addr, np.int32), np.concatenate(fixed)
    m.ndofs = total * components
    m.parts = [dict(elems=np.arange(m.nelem, dtype=np.int32), orient=np.zeros(m.nelem, np.int32), norient=1, weights=weights,
                    lagrange=lagrange, tables=tab[:, None], addr=[(addr + c * total).astype(np.int32) for c in range(components)])]
    m.constrained = np.zeros(m.ndofs, np.uint8)
    for c in range(components):
        m.constrained[fixed + c * total] = 1
    return m


def _tets(n, order, components, kind, mixed):
    """Cubes cut in six tetrahedra with shuffled local vertices; functions numbered by component, then entity.

    kind "h1" (order or, mixed, orders 1 .. order per element) or "curl".  An
    entity carries the functions of the lowest order around it; the others of
    an element have no address there (-1)."""
    m = _Mesh()
    m.dim, m.type, m.components = 3, TET, components
    rng = np.random.Generator(np.random.PCG64(1000 * n + order))
    idx = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij")).reshape(3, -1)[::-1]
    stride = np.array([1, n + 1, (n + 1) ** 2])
    tets = []
    for perm in itertools.permutations(range(3)):
        corner, verts = np.zeros(3, int), [np.zeros(3, int)]
        for a in perm:
            corner = corner.copy()
            corner[a] = 1
            verts.append(corner)
        tets.append(np.stack([((idx + v[:, None]) * stride[:, None]).sum(0) for v in verts], axis=1))
    conn = np.stack(tets, axis=1).reshape(-1, 4)
    conn = rng.permuted(conn, axis=1)
    m.conn, m.nelem = np.ascontiguousarray(conn, np.int32), len(conn)
    nodes = np.stack(np.meshgrid(*[np.arange(n + 1)] * 3, indexing="ij")).reshape(3, -1)[::-1]
    m.grid, m.h = nodes.T / n, 1.0 / n
    rank = np.argsort(conn, axis=1)  # k-th smallest vertex is local vertex rank[:, k]
    srt = np.take_along_axis(conn, rank, axis=1).astype(np.int64)
    code = np.array([sum(p[k] * 4 ** k for k in range(4)) for p in PERMS])
    lookup = np.zeros(256, np.int32)
    lookup[code] = np.arange(24)
    orient = lookup[(rank * 4 ** np.arange(4)).sum(1)]
    orders = rng.integers(1, order + 1, m.nelem) if mixed else np.full(m.nelem, order)
    m.orders = orders
    nn = int((n + 1) ** 3)

    def entities(which):
        keys = np.zeros((m.nelem, len(which)), np.int64)
        for c, vs in enumerate(which):
            for v in vs:
                keys[:, c] = keys[:, c] * nn + srt[:, v]
        u, inv = np.unique(keys, return_inverse=True)
        return u, inv.reshape(m.nelem, len(which))

    ek, ei = entities(EDGES)
    fk, fi = entities(FACES)
    elem_entities = {"v": srt, "e": ei, "f": fi, "c": np.arange(m.nelem)[:, None]}
    count = {"v": nn, "e": len(ek), "f": len(fk), "c": m.nelem}
    low = {}
    for k in "vefc":
        low[k] = np.full(count[k], 99)
        np.minimum.at(low[k], elem_entities[k].ravel(), np.repeat(orders, elem_entities[k].shape[1]))

    def functions(k, p):
        if kind == "curl":
            return {"v": 0 * p, "e": np.minimum(p, 2), "f": np.where(p > 1, 2, 0), "c": 0 * p}[k]
        q = np.maximum
        return {"v": 0 * p + 1, "e": q(p - 1, 0), "f": q(p - 1, 0) * q(p - 2, 0) // 2, "c": q(p - 1, 0) * q(p - 2, 0) * q(p - 3, 0) // 6}[k]

    base, have, total = {}, {}, 0
    for k in "vefc":
        have[k] = functions(k, low[k])
        base[k] = total + np.concatenate([[0], np.cumsum(have[k])])[:-1]
        total += int(have[k].sum())
    m.ndofs = total * components
    m.have, m.elem_entities, m.count = have, elem_entities, count

    def address(k, c, num, sel):
        ent = elem_entities[k][sel, c]
        return np.where(num < have[k][ent], base[k][ent] + num, -1)

    m.parts = []
    for p in sorted(set(orders.tolist())):
        sel = np.flatnonzero(orders == p)
        sel = sel[np.argsort(orient[sel], kind="stable")]
        lam, weights = _tet_points(p + 1)
        if kind == "curl":
            tab = np.stack([_tet_curl_tables(p, lam, perm) for perm in PERMS], axis=1)
            rows = [("e", e, k) for e in range(6) for k in range(min(p, 2))] + ([("f", f, k) for f in range(4) for k in range(2)] if p > 1 else [])
        else:
            tab = np.stack([_tet_h1_tables(p, lam, perm) for perm in PERMS], axis=1)
            rows = [f[:3] for f in _tet_h1(lam, p)]
        addr = np.array([address(k, c, num, sel) for k, c, num in rows], np.int32)
        lag = np.concatenate([lam[None], np.repeat(GRAD.T[:, :, None], lam.shape[1], axis=2)])
        m.parts.append(dict(elems=sel.astype(np.int32), orient=orient[sel].astype(np.int32), norient=24, weights=weights, lagrange=lag, tables=tab,
                            addr=[np.where(addr >= 0, addr + c * total, -1).astype(np.int32) for c in range(components)]))
    m.constrained = np.zeros(m.ndofs, np.uint8)
    bottom = nodes[2] == 0
    side = bottom if components > 1 else ((nodes == 0) | (nodes == n)).any(0)
    fixed = []
    for k, keys in (("v", np.arange(nn)), ("e", ek), ("f", fk)):
        vs = np.stack([keys // nn ** j % nn for j in range({"v": 1, "e": 2, "f": 3}[k])])
        on = side[vs].all(0) if k == "v" else _common_side(nodes, vs, n, bottom_only=components > 1)
        for num in range(int(have[k].max(initial=0))):
            fixed.append((base[k] + num)[on & (num < have[k])])
    fixed = np.concatenate(fixed).astype(np.int64)
    for c in range(components):
        m.constrained[fixed + c * total] = 1
    return m


def _common_side(nodes, vs, n, bottom_only):
    """Whether the vertices of each entity lie on one common side of the cube (the side z = 0 alone)."""
    on = (nodes[2][vs] == 0).all(0)
    if not bottom_only:
        for a in range(3):
            on |= (nodes[a][vs] == 0).all(0) | (nodes[a][vs] == n).all(0)
    return on


_meshes = {}


def _mesh(case):
    key = (case["problem"], case["cell"], case["order"], case["n"])
    if key not in _meshes:
        components = 3 if case["problem"] == "elasticity" else 1
        if case["cell"] == "tet":
            m = _tets(case["n"], case["order"], components, "curl" if case["problem"] == "eddy" else "h1", case["problem"] == "helmholtz")
            if case["problem"] == "eddy":  # two harmonics of one field
                for p in m.parts:
                    a = p["addr"][0]
                    p["addr"] = [a, np.where(a >= 0, a + m.ndofs, -1).astype(np.int32)]
                m.constrained = np.concatenate([m.constrained] * 2)
                m.ndofs *= 2
        else:
            m = _grid(2 if case["cell"] == "quad" else 3, case["n"], case["order"], components)
        if len(_meshes) >= BURST_TEMPLATES:
            _meshes.pop(next(iter(_meshes)))
        _meshes[key] = m
    return _meshes[key]


# ---------------------------------------------------------------- weak forms

class _Program:
    """Coefficient program with shared subexpressions."""

    def __init__(self):
        self.nodes, self.consts, self.seen = [], [], {}

    def node(self, op, a=0, b=0):
        k = (op, a, b)
        if k not in self.seen:
            self.seen[k] = len(self.nodes)
            self.nodes.append((op, a, b, 0))
        return self.seen[k]

    def const(self, v):
        if v not in self.consts:
            self.consts.append(v)
        return self.node(abi.OP_CONST, self.consts.index(v))

    def mul(self, *xs):
        r = xs[0]
        for x in xs[1:]:
            r = self.node(abi.OP_MUL, r, x)
        return r

    def add(self, *xs):
        r = xs[0]
        for x in xs[1:]:
            r = self.node(abi.OP_ADD, r, x)
        return r

    def inv(self, k, a):
        return self.node(abi.OP_INVJAC, k, a)


def _forms(case, m, part, rng):
    """Groups of one element set: dicts of GroupBuilder arguments with the arrays the seed decides."""
    dim, T = m.dim, part["tables"]
    ntab, rows = len(T), T.shape[2]
    data = [rng.lognormal(0.0, 0.5, part["elems"].size)]
    common = dict(elemtype=m.type, dim=dim, elems=part["elems"], orient=part["orient"], norient=part["norient"], weights=part["weights"],
                  lagrange=part["lagrange"], ncurvednodes=m.conn.shape[1], ntf=rows, ndof=rows, tables=[T[k] for k in range(ntab)])
    pairs = [(a, b) for a in range(dim) for b in range(dim)]
    if case["problem"] == "elasticity":
        out = []
        for i, j in itertools.product(range(3), repeat=2):
            P = _Program()
            E = P.node(abi.OP_ELEM, 0)
            lam, mu = P.mul(E, P.const(0.3 / (1.3 * 0.4))), P.mul(E, P.const(0.5 / 1.3))
            terms = []
            for a, b in pairs:
                c = P.add(P.mul(lam, P.inv(i, a), P.inv(j, b)), P.mul(mu, P.inv(j, a), P.inv(i, b)))
                if i == j:
                    c = P.add(c, P.mul(mu, P.add(*[P.mul(P.inv(k, a), P.inv(k, b)) for k in range(3)])))
                terms.append((1 + a, 1 + b, c, 1.0))
            out.append(dict(common, nodes=P.nodes, consts=P.consts, terms=terms, elemdata=data,
                            dests=[(part["addr"][i], part["addr"][j], 1.0)]))
        return out
    if case["problem"] == "eddy":
        mass, curl = _Program(), _Program()
        s = mass.node(abi.OP_ELEM, 0)
        mt = [(a, b, mass.mul(s, mass.add(*[mass.mul(mass.inv(k, a), mass.inv(k, b)) for k in range(3)])), 1.0) for a, b in pairs]
        det = curl.node(abi.OP_DETJAC)
        w = curl.mul(curl.const(1 / (4e-7 * math.pi)), curl.node(abi.OP_INV, curl.mul(det, det)))
        jac = lambda a, k: curl.node(abi.OP_JAC, a, k)  # noqa: E731
        ct = [(3 + a, 3 + b, curl.mul(w, curl.add(*[curl.mul(jac(a, k), jac(b, k)) for k in range(3)])), 1.0) for a, b in pairs]
        u2, u3 = part["addr"]
        sigma = [np.array([1e3, 5.0e5, 2.0e6, 6.0e7])[rng.integers(0, 4, part["elems"].size)]]
        return [dict(common, nodes=curl.nodes, consts=curl.consts, terms=ct, elemdata=[], dests=[(u2, u2, 1.0), (u3, u3, 1.0)]),
                dict(common, nodes=mass.nodes, consts=[], terms=mt, elemdata=sigma, dests=[(u2, u3, 1.0), (u3, u2, -1.0)])]
    P = _Program()
    k = P.node(abi.OP_ELEM, 0)
    terms = [(1 + a, 1 + b, P.mul(k, P.add(*[P.mul(P.inv(d, a), P.inv(d, b)) for d in range(dim)])), 1.0) for a, b in pairs]
    if case["problem"] == "helmholtz":
        terms.append((0, 0, P.mul(k, P.const(-25.0)), 1.0))
    return [dict(common, nodes=P.nodes, consts=P.consts, terms=terms, elemdata=data, dests=[(part["addr"][0], part["addr"][0], 1.0)])]


def _source(m, part, rng):
    """Right-hand side of a source interpolated with the field's own functions."""
    T = part["tables"]
    rows = T.shape[2]
    return dict(elemtype=m.type, dim=m.dim, elems=part["elems"], orient=part["orient"], norient=1, weights=part["weights"],
                lagrange=part["lagrange"], ncurvednodes=m.conn.shape[1], ntf=rows, ndof=1, tables=[T[0]],
                nodes=[(abi.OP_FIELD, 0, 0, 0)], consts=[], terms=[(0, -1, 0, 1.0)], dests=[(part["addr"][0], None, 1.0)],
                fielddata=[rng.standard_normal((rows, part["elems"].size))])


def _problem(case, seed):
    m = _mesh(case)
    rng = np.random.Generator(np.random.PCG64(seed))
    xyz = np.zeros((len(m.grid), 3))
    xyz[:, :m.dim] = m.grid
    inner = ((m.grid > 1e-9) & (m.grid < 1 - 1e-9)).all(1)
    xyz[inner, :m.dim] += rng.uniform(-0.15, 0.15, (int(inner.sum()), m.dim)) * m.h
    if case["call"] == "rhs":
        return m, xyz, [_source(m, p, rng) for p in m.parts]
    return m, xyz, [g for p in m.parts for g in _forms(case, m, p, rng)]


def _sweep_scales(seed, nterms):
    """Term scales of the eddy problem's two groups at one angular frequency."""
    w = 2 * math.pi * 10.0 ** np.random.Generator(np.random.PCG64(seed + 77)).uniform(0, 6)
    return [np.ones(nterms), np.full(nterms, w)]


def _renumbered(m, groups, seed, count=12):
    """The groups and constraints with the DOF numbers shifted cyclically, by another amount each: the numbering of a
    program that added fields or adapted its mesh in between."""
    rng = np.random.Generator(np.random.PCG64(seed + 5))
    out = []
    for _ in range(count):
        by, done = int(rng.integers(1, m.ndofs)), {}

        def shifted(a):
            if id(a) not in done:  # the groups share their address arrays
                done[id(a)] = np.where(a >= 0, (a + by) % m.ndofs, -1).astype(np.int32)
            return done[id(a)]

        out.append(([dict(g, dests=[(shifted(tf), shifted(dof), mult) for tf, dof, mult in g["dests"]]) for g in groups],
                    np.roll(m.constrained, by)))
    return out


# ---------------------------------------------------------------- one program's use of the engine

_context = None
_numbers = itertools.count(1)


def _ctx():
    global _context
    if _context is None:
        _context = abi.Context(0)
        _context.check(_context.lib.slgpu_ctx_set_kernel_timers(_context.h, 0))
    return _context


class _Borrowed:
    """Numbers that the engine owns, on the device or page-locked, for a view without a copy; keeps their owner."""

    def __init__(self, owner, ptr, n, device, kind="<f8"):
        self.owner = owner
        setattr(self, "__cuda_array_interface__" if device else "__array_interface__",
                dict(shape=(n,), typestr=kind, data=(ptr, False), version=2 if device else 3))


def _on_device(owner, ptr, n, kind="<f8"):
    if n == 0:
        return torch.empty(0, dtype=torch.float64 if kind == "<f8" else torch.int32, device="cuda")
    return torch.as_tensor(_Borrowed(owner, ptr.value, n, True, kind), device="cuda")


def _on_host(owner, pinned, n):
    return np.asarray(_Borrowed(owner, pinned.ptr.value, n, False))


class _State:
    def __init__(self, case, seed):
        self.case, self.handles, self.server, self.pinned = case, [], None, []
        self.ctx = _ctx() if case["call"] != "serve" else abi.Context(0)
        self.lib, self.at = self.ctx.lib, 0
        self.precision = PRECISION[case["precision"]]

    def mesh(self, m, xyz):
        number = next(_numbers) % 64  # a few meshes stay resident, older numbers are taken again
        self.ctx.check(self.lib.slgpu_mesh_set_nodes(self.ctx.h, number, len(xyz), abi.f64p(xyz)))
        self.ctx.check(self.lib.slgpu_mesh_set_elements(self.ctx.h, number, m.type, m.conn.shape[1], m.nelem, abi.i32p(m.conn)))
        return number

    def matrix(self, ndofs, groups):
        h = ctypes.c_int()
        self.ctx.check(self.lib.slgpu_matrix_create(self.ctx.h, ndofs, ctypes.byref(h)))
        self.ctx.check(self.lib.slgpu_matrix_share_addresses(self.ctx.h, h, 1))
        for g in groups:
            self.ctx.check(self.lib.slgpu_matrix_add_group(self.ctx.h, h, ctypes.byref(g.g), None))
        return h.value

    def process(self, h, constrained):
        info = abi.CsrInfo()
        self.ctx.check(self.lib.slgpu_matrix_process(self.ctx.h, h, constrained.ctypes.data_as(POINTER(c_uint8)), self.precision, ctypes.byref(info)))
        return info

    def close(self):
        if self.server is not None:
            self.server.close()
            self.server = None
        for p in self.pinned:
            p.close()
        for h in self.handles:
            self.lib.slgpu_matrix_destroy(self.ctx.h, h)
        self.handles, self.pinned = [], []

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def _builders(groups, number):
    return [abi.GroupBuilder(mesh=number, **g) for g in groups]


def prepare(case, seed):
    s = _State(case, seed)
    if case["call"] == "serve":
        return _prepare_serve(s, seed)
    m, xyz, groups = _problem(case, seed)
    s.m, s.ndofs = m, m.ndofs
    number = s.mesh(m, xyz)
    s.groups = _builders(groups, number)
    s.constrained = m.constrained
    if case["call"] == "rhs":
        n = sum(g.g.ntf * g.g.nelem for g in s.groups)
        s.rows, s.vals = np.zeros(n, np.int32), np.zeros(n)
        return s
    if case["call"] == "first":
        s.numberings = [(_builders(g, number), con) for g, con in _renumbered(m, groups, seed)]
        return s
    h = s.matrix(s.ndofs, s.groups)
    s.handles.append(h)
    s.info = s.process(h, s.constrained)
    if case["call"] == "generate":
        s.pinned = [serving.PinnedArray(s.lib, s.ctx.h, max(1, v)) for v in (s.info.nnzA, s.info.nnzD)]
        return s
    s.scales = _sweep_scales(seed, len(groups[0]["terms"])) if case["call"] == "sweep" else None
    # One array per element set, as a program holds its material field.
    s.fields = [(i, np.ascontiguousarray(g["elemdata"][0])) for i, g in enumerate(groups) if g["elemdata"]] if case["data"] == "element" else []
    s.b = torch.randn(s.ndofs, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed)) if case["eliminate"] else None
    s.ba = torch.empty(s.info.nA, dtype=torch.float64, device="cuda") if case["eliminate"] else None
    s.groups = None
    torch.cuda.synchronize()
    return s


def _serve_pool(case):
    """The burst's templates: problems of four kinds scaled by n."""
    n = case["n"]
    mk = lambda p, c, o, k: _case("", "step", p, c, o, k, case["precision"])  # noqa: E731
    return [mk("poisson", "quad", 1, 20 * n), mk("poisson", "quad", 3, 5 * n), mk("elasticity", "hex", 2, n), mk("poisson", "tet", 2, n)]


def _prepare_serve(s, seed):
    case = s.case
    s.ctx.check(s.lib.slgpu_ctx_set_kernel_timers(s.ctx.h, 0))
    s.templates = []
    for k, c in enumerate(_serve_pool(case)):
        m, xyz, groups = _problem(c, seed + k)
        h = s.matrix(m.ndofs, _builders(groups, s.mesh(m, xyz)))
        s.handles.append(h)
        s.templates.append((h, s.process(h, m.constrained), len(groups), m.nelem))
    s.server = serving.Server(s.lib, s.ctx.h, 4)
    for h, _, _, _ in s.templates:
        s.server.prepare(h, s.precision)
    s.requests = []
    rng = np.random.Generator(np.random.PCG64(seed + 900))
    for r in range(case["requests"]):
        h, info, ngroups, nelem = s.templates[r % BURST_TEMPLATES]
        field, A, D = (serving.PinnedArray(s.lib, s.ctx.h, max(1, k)) for k in (nelem, info.nnzA, info.nnzD))
        s.pinned += [field, A, D]
        field.array[:] = rng.lognormal(0.0, 0.5, nelem)
        updates = [serving.UpdateSpec(g, abi.UPDATE_ELEMDATA, 0, field.array) for g in range(ngroups)]
        s.requests.append((h, info, updates, A, D))
    return s


def run(s):
    return {"step": _run_step, "sweep": _run_step, "generate": _run_generate, "first": _run_first, "rhs": _run_rhs, "serve": _run_serve}[s.case["call"]](s)


def _device_csr(s, h, info, structure=True):
    p = [c_void_p() for _ in range(6)]
    s.ctx.check(s.lib.slgpu_matrix_device_csr(s.ctx.h, h, *[ctypes.byref(q) for q in p]))
    out = {"A": _on_device(s, p[2], info.nnzA), "D": _on_device(s, p[5], info.nnzD)}
    if structure:
        for name, q, n in (("Arows", p[0], info.nA + 1), ("Acols", p[1], info.nnzA), ("Drows", p[3], info.nA + 1), ("Dcols", p[4], info.nnzD)):
            out[name] = _on_device(s, q, n, "<i4")
    return out


def _run_step(s):
    h = s.handles[0]
    for gi, e in s.fields:
        s.ctx.check(s.lib.slgpu_matrix_set_elemdata(s.ctx.h, h, gi, 0, abi.f64p(e)))
    if s.scales is not None:
        for gi, v in enumerate(s.scales):
            s.ctx.check(s.lib.slgpu_matrix_set_scales(s.ctx.h, h, gi, abi.f64p(v), None))
    info = s.process(h, s.constrained)
    out = _device_csr(s, h, info, structure=False)
    if s.b is not None:
        s.ctx.check(s.lib.slgpu_matrix_eliminate(s.ctx.h, h, c_void_p(s.b.data_ptr()), c_void_p(s.ba.data_ptr())))
        out["ba"] = s.ba
    return out


def _run_generate(s):
    h = s.matrix(s.ndofs, s.groups)
    info = s.process(h, s.constrained)
    A, D = s.pinned
    s.ctx.check(s.lib.slgpu_matrix_download_values(s.ctx.h, h, abi.f64p(A.array), abi.f64p(D.array)))
    s.ctx.check(s.lib.slgpu_matrix_destroy(s.ctx.h, h))
    return {"A": _on_host(s, A, info.nnzA), "D": _on_host(s, D, info.nnzD)}


def _run_first(s):
    groups, constrained = s.numberings[s.at % len(s.numberings)]
    s.at += 1
    for old in s.handles:
        s.ctx.check(s.lib.slgpu_matrix_destroy(s.ctx.h, old))
    s.handles = [s.matrix(s.ndofs, groups)]
    info = s.process(s.handles[0], constrained)
    return _device_csr(s, s.handles[0], info)


def _run_rhs(s):
    out = {}
    for k, g in enumerate(s.groups):
        count = c_int64()
        s.ctx.check(s.lib.slgpu_rhs_assemble_rows(s.ctx.h, ctypes.byref(g.g), s.ndofs, s.precision, abi.i32p(s.rows), abi.f64p(s.vals),
                                                  s.rows.size, ctypes.byref(count)))
        out["rows%d" % k], out["vals%d" % k] = s.rows[: count.value], s.vals[: count.value]
    return out


def _run_serve(s):
    tickets = [s.server.submit(h, s.precision, updates, A.array, D.array[: info.nnzD]) for h, info, updates, A, D in s.requests]
    for t in tickets:
        s.server.wait(t)
    return {"%d" % k: {"A": _on_host(s, A, info.nnzA), "D": _on_host(s, D, info.nnzD)} for k, (_, info, _, A, D) in enumerate(s.requests)}


# ---------------------------------------------------------------- work and exact values

def _nnz(m):
    """CSR entries of the field's DOFs coupled inside elements (before the rows of constrained ones are dropped)."""
    if hasattr(m, "have"):
        cols = np.concatenate([m.elem_entities[k] + o for k, o in zip("vefc", np.cumsum([0] + [m.count[k] for k in "vef"]))], axis=1)
        have = np.concatenate([m.have[k] for k in "vefc"]).astype(np.int64)
        keys = np.unique((cols[:, :, None].astype(np.int64) * have.size + cols[:, None, :]).ravel())
        scalar = int((have[keys // have.size] * have[keys % have.size]).sum())
        return scalar * m.components ** 2
    n = round(1 / m.h)
    p = round(m.parts[0]["tables"].shape[2] ** (1 / m.dim)) - 1
    line = (3 * n + 1) + 2 * (p - 1) * 2 * n + (p - 1) ** 2 * n
    return line ** m.dim * m.components ** 2


def work(case):
    """Bytes: mesh, coefficients and addresses read, CSR values (and what else comes back) written.  FLOPs: the element
    contraction of every distinct entry (upper triangles of symmetric blocks, one of each transposed pair)."""
    if case["call"] == "serve":
        total = {"bytes": 0.0, "flops": 0.0}
        for r in range(case["requests"]):
            w = work(_serve_pool(case)[r % BURST_TEMPLATES])
            total = {k: total[k] + w[k] for k in total}
        return total
    m, _, groups = _problem(case, 1)
    nbytes = m.grid.shape[0] * 24.0 + m.conn.size * 4.0 + sum(4.0 * a.size for p in m.parts for a in p["addr"])
    flops = 0.0
    for g in groups:
        e, P = g["elems"].size, g["ntf"] * g["ndof"]
        distinct = P if case["call"] == "rhs" else (P + g["ntf"]) / 2
        if case["problem"] == "elasticity":  # per group: three symmetric blocks and three transposed pairs over nine
            distinct = (3 * (P + g["ntf"]) / 2 + 3 * P) / 9
        flops += 2.0 * distinct * len(g["terms"]) * len(g["weights"]) * e
    for p in m.parts:
        nbytes += 8.0 * p["elems"].size
    if case["call"] == "rhs":
        return {"bytes": nbytes + sum(8.0 * f.size for g in groups for f in g["fielddata"]) + 12.0 * m.ndofs, "flops": flops}
    nnz = _nnz(m) * (4 if case["problem"] == "eddy" else 1)
    return {"bytes": nbytes + (12.0 if case["call"] == "first" else 8.0) * nnz, "flops": flops}


def _coefficients(g, m, xyz, data):
    """[terms][elements, points]: coefficient times weight times |det J|, in torch."""
    dev = "cuda"
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
    X = t(xyz)[t(m.conn.astype(np.int64))[t(g["elems"].astype(np.int64))]][:, :, : m.dim]
    lag = t(g["lagrange"])
    J = torch.einsum("akg,ekx->egax", lag[1:], X)
    det, inv = torch.linalg.det(J), torch.linalg.inv(J)
    vals = []
    for op, a, b, _ in g["nodes"]:
        if op == abi.OP_CONST:
            v = torch.full_like(det, g["consts"][a])
        elif op == abi.OP_JAC:
            v = J[:, :, a, b]
        elif op == abi.OP_INVJAC:
            v = inv[:, :, a, b]
        elif op == abi.OP_DETJAC:
            v = det
        elif op == abi.OP_ELEM:
            v = t(data[a])[:, None].expand_as(det)
        elif op == abi.OP_FIELD:
            v = torch.einsum("re,rg->eg", t(g["fielddata"][a]), t(g["tables"][b])[0])
        elif op == abi.OP_ADD:
            v = vals[a] + vals[b]
        elif op == abi.OP_MUL:
            v = vals[a] * vals[b]
        else:
            v = 1.0 / vals[a]
        vals.append(v)
    w = det.abs() * t(g["weights"])
    return [vals[c] * scale * w for _, _, c, scale in g["terms"]]


def _element_matrices(g, m, xyz, data, scales):
    """[elements, ntf * ndof], orientation by orientation."""
    C = _coefficients(g, m, xyz, data)
    if scales is not None:
        C = [c * s for c, s in zip(C, scales)]
    tab = [torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in g["tables"]]
    V = torch.empty(g["elems"].size, g["ntf"] * g["ndof"], dtype=torch.float64, device="cuda")
    orient = torch.as_tensor(g["orient"].astype(np.int64), device="cuda")
    for o in torch.unique(orient).tolist():
        sel = (orient == o).nonzero()[:, 0]
        acc = 0
        for (tf, dof, _, _), c in zip(g["terms"], C):
            M = tab[tf][o] if dof < 0 else (tab[tf][o][:, None] * tab[dof][o][None]).reshape(V.shape[1], -1)
            acc = acc + c[sel] @ M.T
        V[sel] = acc
    return V


def _assembled(case, m, xyz, groups, constrained, scales=None, data=None):
    """A and D (rows, columns, values) in 64 bits."""
    n = m.ndofs
    con = torch.as_tensor(constrained, device="cuda").bool()
    local = torch.where(con, torch.cumsum(con, 0) - 1, torch.cumsum(~con, 0) - 1)
    keys, vals = [], []
    for gi, g in enumerate(groups):
        V = _element_matrices(g, m, xyz, g["elemdata"] if data is None else [data], None if scales is None else scales[gi])
        for tf, dof, mult in g["dests"]:
            r = torch.as_tensor(tf.astype(np.int64), device="cuda").T[:, :, None]
            c = torch.as_tensor(dof.astype(np.int64), device="cuda").T[:, None, :]
            ok = ((r >= 0) & (c >= 0) & ~con[r.clamp(min=0)]).reshape(-1)
            keys.append((r * n + c).reshape(-1)[ok])
            vals.append(V.reshape(-1)[ok] * mult)
    keys, vals = torch.cat(keys), torch.cat(vals)
    srt, perm = torch.sort(keys)
    del keys
    uniq, inverse = torch.unique_consecutive(srt, return_inverse=True)
    del srt
    total = torch.zeros(uniq.numel(), dtype=torch.float64, device="cuda").index_add_(0, inverse, vals[perm])
    del inverse, perm, vals
    row, col = local[uniq // n], uniq % n
    in_d = con[col]
    nA = int((~con).sum())

    def block(sel):
        ptr = torch.zeros(nA + 1, dtype=torch.int64, device="cuda")
        ptr[1:] = torch.cumsum(torch.bincount(row[sel], minlength=nA), 0)
        return ptr.int(), local[col[sel]].int(), total[sel]

    return block(~in_d), block(in_d)


def exact(case, seed):
    if case["call"] == "serve":
        out, rng, pool = {}, np.random.Generator(np.random.PCG64(seed + 900)), _serve_pool(case)
        problems = []
        for k, c in enumerate(pool):
            m, xyz, groups = _problem(c, seed + k)
            problems.append((m, xyz, groups))
        for r in range(case["requests"]):
            m, xyz, groups = problems[r % BURST_TEMPLATES]
            field = rng.lognormal(0.0, 0.5, m.nelem)
            # Requests carry fields in mesh element order; a group holds its elements in its own.
            A, D = _assembled(pool[r % BURST_TEMPLATES], m, xyz, groups, m.constrained, data=field[groups[0]["elems"]])
            out["%d" % r] = {"A": A[2], "D": D[2]}
        return out
    m, xyz, groups = _problem(case, seed)
    if case["call"] == "rhs":
        out = {}
        for k, g in enumerate(groups):
            V = _element_matrices(g, m, xyz, [], None)
            a = torch.as_tensor(g["dests"][0][0].astype(np.int64), device="cuda").T.reshape(-1)
            total = torch.zeros(m.ndofs, dtype=torch.float64, device="cuda").index_add_(0, a, -V.reshape(-1))
            rows = torch.unique(a)
            out["rows%d" % k], out["vals%d" % k] = rows.int(), total[rows]
        return out
    constrained = m.constrained
    if case["call"] == "first":
        groups, constrained = _renumbered(m, groups, seed)[0]
    scales = _sweep_scales(seed, len(groups[0]["terms"])) if case["call"] == "sweep" else None
    A, D = _assembled(case, m, xyz, groups, constrained, scales)
    if case["call"] == "first":
        return {"Arows": A[0], "Acols": A[1], "A": A[2], "Drows": D[0], "Dcols": D[1], "D": D[2]}
    out = {"A": A[2], "D": D[2]}
    if case["eliminate"]:
        b = torch.randn(m.ndofs, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
        con = torch.as_tensor(m.constrained, device="cuda").bool()
        bd = b[con][D[1].long()] * D[2]
        row = torch.repeat_interleave(torch.arange(D[0].numel() - 1, device="cuda"), (D[0][1:] - D[0][:-1]).long())
        out["ba"] = b[~con] - torch.zeros(D[0].numel() - 1, dtype=torch.float64, device="cuda").index_add_(0, row, bd)
    return out
