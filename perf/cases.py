"""The work a user has the geometry path do, as cases with inputs of their own.

A case is one of six kinds of call, on a mesh built on the GPU from the seed (sin-mapped boxes and
a torus, interior nodes jittered):

- ``evaluate``: one block's factors in one fused launch, the call an assembly loop makes, in the
  mesh's own type ("native": f64 or f32), double-float ("df64") or split precision, with the
  measure of the block where the case asks for it;
- ``batch``: every block of a hybrid mesh in one graph launch;
- ``vjp``: one block's forward factors and node cotangents in one call;
- ``adjoint_batch``: forward and adjoint of a hybrid mesh in one graph launch;
- ``pull_back``: reference coordinates of points given in physical space, cell by cell.

``exact`` restates every result in 64-bit torch from the lattice the meshes are built on: monomial
expansions with exactly rational coefficients, cofactors, and automatic differentiation for the
adjoint.
"""

from __future__ import annotations

import fractions
import functools
import math

import numpy as np
import torch

import gridcl_gb300 as tg

DEV = "cuda"
TILE = 16
TDIM = {"Triangle": 2, "Tetrahedron": 3, "Hexahedron": 3, "Prism": 3}
FACTORS = {
    "all": ("points", "jacobian", "detj", "pinv"),  # what a general form needs
    "assembly": ("detj", "pinv"),  # a Laplacian's
    "surface": ("points", "detj", "normals"),  # a flux or boundary-element integral's
}
LEN = {"points": lambda td: 3, "jacobian": lambda td: 3 * td, "detj": lambda td: 1, "pinv": lambda td: 3 * td,
       "normals": lambda td: 3}


def listed():
    return [
        # A unit test's or a coarse multigrid level's mesh: a call is launch and host time.
        {"name": "p1_tets_small_f64", "kind": "evaluate", "cell": "Tetrahedron", "degree": 1, "cells": 3072,
         "rule": "7x2x1", "precision": "native", "f32": False, "factors": "all", "measure": False},
        # Curved tetrahedra, 1.5 million cells: the default precision, ...
        {"name": "p2_tets_f64", "kind": "evaluate", "cell": "Tetrahedron", "degree": 2, "cells": 1572864,
         "rule": "4x3x2", "precision": "native", "f32": False, "factors": "all", "measure": False},
        # ... the f64-accurate path on the FP32 pipe, ...
        {"name": "p2_tets_df64", "kind": "evaluate", "cell": "Tetrahedron", "degree": 2, "cells": 1572864,
         "rule": "4x3x2", "precision": "df64", "f32": False, "factors": "all", "measure": False},
        # ... and a single-precision step that also takes the mesh's volume.
        {"name": "p2_tets_split_measure", "kind": "evaluate", "cell": "Tetrahedron", "degree": 2, "cells": 1572864,
         "rule": "4x3x2", "precision": "split", "f32": False, "factors": "all", "measure": True},
        # Triquadratic hexahedra at the Gauss rule, a cell count that is no multiple of a tile.
        {"name": "q2_hexes_f64", "kind": "evaluate", "cell": "Hexahedron", "degree": 2, "cells": 226981,
         "rule": "3x3x3", "precision": "native", "f32": False, "factors": "all", "measure": False},
        # A closed surface of high-order triangles: area elements and normals of boundary integrals.
        {"name": "p4_surface_split", "kind": "evaluate", "cell": "Triangle", "degree": 4, "cells": 1048583,
         "rule": "7x4", "precision": "split", "f32": False, "factors": "surface", "measure": False},
        # High-order tetrahedra of a spectral code on a single-precision mesh.
        {"name": "p5_tets_f32", "kind": "evaluate", "cell": "Tetrahedron", "degree": 5, "cells": 24576,
         "rule": "6x6x6", "precision": "native", "f32": True, "factors": "all", "measure": False},
        # A large hybrid mesh, every block in one launch: f64-accurate forward, ...
        {"name": "hybrid_forward_df64", "kind": "batch", "hexes": 2000000, "prisms": 300000, "tets": 50000,
         "precision": "df64"},
        # ... and a shape-optimisation step: forward and node cotangents in split precision.
        {"name": "hybrid_adjoint_split", "kind": "adjoint_batch", "hexes": 2000000, "prisms": 300000, "tets": 50000,
         "precision": "split"},
        # One block's forward and adjoint in the default precision (a mesh-smoothing step).
        {"name": "q2_hexes_adjoint_f64", "kind": "vjp", "cell": "Hexahedron", "degree": 2, "cells": 110592,
         "rule": "3x3x3", "precision": "native"},
        # Points to reference coordinates (interpolation between meshes, particles): f64, ...
        {"name": "pull_back_p2_tets_f64", "kind": "pull_back", "cell": "Tetrahedron", "degree": 2, "cells": 48000,
         "points": 24, "precision": "native", "f32": False},
        # ... and mixed precision on hexahedra.
        {"name": "pull_back_q2_hexes_split", "kind": "pull_back", "cell": "Hexahedron", "degree": 2, "cells": 35937,
         "points": 27, "precision": "split", "f32": False},
    ]


_RULES = {("Tetrahedron", 1): ("2x2x2", "7x2x1", "3x3x3"), ("Tetrahedron", 2): ("3x3x3", "4x3x2", "4x4x4"),
          ("Tetrahedron", 3): ("4x4x4", "4x3x2"), ("Hexahedron", 1): ("2x2x2", "3x3x3"),
          ("Hexahedron", 2): ("3x3x3", "4x4x4", "3x3x2"), ("Prism", 1): ("2x2x2", "3x1x2"),
          ("Prism", 2): ("3x3x3", "3x1x7"), ("Triangle", 1): ("2x2", "3x2"), ("Triangle", 2): ("3x3", "7x4"),
          ("Triangle", 4): ("7x4", "5x5"), ("Tetrahedron", 4): ("5x5x5",), ("Tetrahedron", 5): ("6x6x6",),
          ("Tetrahedron", 6): ("7x7x7",)}


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], even over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "surface", "high_order", "batch", "adjoint_batch", "vjp", "pull_back"])
    precisions = [("native", False), ("native", True), ("df64", False), ("split", False)]
    if kind in ("evaluate", "surface", "high_order"):
        cell, degree = rng.choice({
            "evaluate": [("Tetrahedron", 1), ("Tetrahedron", 2), ("Tetrahedron", 3), ("Hexahedron", 1),
                         ("Hexahedron", 2), ("Prism", 1), ("Prism", 2)],
            "surface": [("Triangle", 1), ("Triangle", 2), ("Triangle", 4)],
            "high_order": [("Tetrahedron", 4), ("Tetrahedron", 5), ("Tetrahedron", 6)]}[kind])
        precision, f32 = rng.choice(precisions if kind != "high_order" else [("native", True), ("split", False)])
        rule = rng.choice(_RULES[cell, degree])
        most = 12_000_000 // _rule_size(rule)
        measure = kind == "evaluate" and rng.random() < 0.25
        factors = "surface" if kind == "surface" else "all" if measure else rng.choice(["all", "assembly"])
        return {"kind": "evaluate", "cell": cell, "degree": degree, "cells": _spread(rng, 500, most), "rule": rule,
                "precision": precision, "f32": f32, "factors": factors, "measure": measure}
    if kind in ("batch", "adjoint_batch"):
        hexes = _spread(rng, 3000, 500_000)
        return {"kind": kind, "hexes": hexes, "prisms": _spread(rng, 500, 100_000), "tets": _spread(rng, 500, 50_000),
                "precision": rng.choice(["df64", "split"])}
    cell, degree = rng.choice([("Tetrahedron", 1), ("Tetrahedron", 2), ("Hexahedron", 1), ("Hexahedron", 2),
                               ("Prism", 2)])
    if kind == "vjp":
        return {"kind": kind, "cell": cell, "degree": degree, "cells": _spread(rng, 500, 60_000),
                "rule": rng.choice(_RULES[cell, degree]), "precision": rng.choice(["native", "split"])}
    precision, f32 = rng.choice([("native", False), ("native", True), ("split", False)])
    # (In f32 the tolerance of 1e-5 is above the rounding of X only on coarse meshes.)
    return {"kind": kind, "cell": cell, "degree": degree, "cells": _spread(rng, 500, 3_000 if f32 else 30_000),
            "points": rng.choice([4, 8, 15, 24, 27]), "precision": precision, "f32": f32}


# --------------------------------------------------------------------------------------------
# Meshes, on the GPU.

def _rule_size(rule):
    return math.prod(int(c) for c in rule.split("x"))


def _counts(rule):
    return tuple(int(c) for c in rule.split("x"))


def _lattice(cell, p):
    """The nodes of a degree-p cell as lattice points [K][td], lexicographic."""
    r = range(p + 1)
    if cell == "Triangle":
        return np.array([(a, b) for b in r for a in r if a + b <= p])
    if cell == "Tetrahedron":
        return np.array([(a, b, c) for c in r for b in r for a in r if a + b + c <= p])
    if cell == "Prism":
        return np.array([(a, b, c) for c in r for b in r for a in r if a + b <= p])
    return np.array([(a, b, c) for c in r for b in r for a in r])


def _subcell_axes(cell):
    """The cells of one subcell: origin and axis vectors [per][1 + td][dim] in subcell units."""
    bits = np.array([[v & 1, (v >> 1) & 1, (v >> 2) & 1] for v in range(8)])
    if cell == "Triangle":
        return np.array([[[0, 0], [1, 0], [0, 1]], [[1, 1], [-1, 0], [0, -1]]])
    if cell == "Hexahedron":
        sel = [[0, 1, 2, 4]]
    elif cell == "Prism":
        sel = [[0, 1, 3, 4], [0, 3, 2, 4]]
    else:
        sel = []
        for a, b in ((0, 1), (0, 2), (1, 0), (1, 2), (2, 0), (2, 1)):
            v = [0, 1 << a, (1 << a) | (1 << b), 7]
            if np.linalg.det(bits[v[1:]] - bits[0]) < 0:
                v[1], v[2] = v[2], v[1]
            sel.append(v)
    out = []
    for v in sel:
        c = bits[v]
        out.append(np.concatenate([c[:1], c[1:] - c[:1]]))
    return np.array(out)


def _keys(cell, p, cells, local, n):
    """Lattice coordinates [cells][K][dim] of the first `cells` cells' nodes; `local` [K][td] are
    the reference lattice points, `n` the subcells per axis (x fastest)."""
    axes = _subcell_axes(cell)
    per, dim = axes.shape[0], axes.shape[2]
    off = p * axes[:, None, 0] + np.einsum("kt,ptd->pkd", local, axes[:, 1:])
    c = torch.arange(cells, device=DEV)
    sub = c // per
    ijk = [sub % n[0], (sub // n[0]) % n[1]] + ([sub // (n[0] * n[1])] if dim == 3 else [])
    return p * torch.stack(ijk, 1)[:, None, :] + torch.from_numpy(off).to(DEV)[c % per]


def _box(cell, p, cells, seed, amplitude=0.05):
    """Node coordinates [N][3] f64 and the node numbers of a local lattice. Nodes are numbered by
    the first cell that uses them; the jitter is 2 % of a cell's size, less above degree 2, whose
    maps it would fold."""
    jitter = min(0.02, 0.08 / p ** 2)
    per = _subcell_axes(cell).shape[0]
    gen = torch.Generator(device=DEV).manual_seed(seed)
    if cell == "Triangle":  # a torus of 2 nu nv triangles, periodic
        nv = max(3, math.isqrt(max(1, cells // 4)))
        nu = max(3, -(-cells // (2 * nv)))
        shape, n = (nu * p, nv * p), (nu, nv)
    else:
        m = 1
        while per * m ** 3 < cells:
            m += 1
        shape, n = (m * p + 1,) * 3, (m,) * 3
    stride = [1]
    for s in shape[:-1]:
        stride.append(stride[-1] * s)

    def flat(local):
        k = _keys(cell, p, cells, local, n)
        if cell == "Triangle":
            k = torch.remainder(k, torch.tensor(shape, device=DEV))
        return sum(k[..., d] * stride[d] for d in range(len(shape)))

    keys = flat(_lattice(cell, p))
    total = math.prod(shape)
    owner = torch.arange(cells, device=DEV).repeat_interleave(keys.shape[1])
    first = torch.full((total,), cells, device=DEV).scatter_reduce_(0, keys.reshape(-1), owner, "amin")
    used = torch.nonzero(first < cells).reshape(-1)
    used = used[torch.argsort(first[used], stable=True)]
    number = torch.full((total,), -1, dtype=torch.int64, device=DEV)
    number[used] = torch.arange(used.numel(), device=DEV)
    at = torch.stack([(used // stride[d]) % shape[d] for d in range(len(shape))], 1).double()
    noise = 2.0 * torch.rand((total, 3), generator=gen, dtype=torch.float64, device=DEV)[used] - 1.0
    if cell == "Triangle":
        ph = 2.0 * math.pi * torch.rand(2, generator=gen, dtype=torch.float64, device=DEV)
        u, v = (2.0 * math.pi * at[:, d] / shape[d] for d in range(2))
        r = 0.4 * (1.0 + amplitude * torch.sin(3.0 * u + ph[0]) * torch.sin(2.0 * v + ph[1]))
        r = r * (1.0 + jitter * 2.0 * math.pi / n[1] * noise[:, 0] / p)
        x = torch.stack([(1.0 + r * torch.cos(v)) * torch.cos(u), (1.0 + r * torch.cos(v)) * torch.sin(u),
                         r * torch.sin(v)], 1)
    else:
        x = at / (shape[0] - 1)
        inner = ((at > 0) & (at < shape[0] - 1)).all(1, keepdim=True)
        s = torch.sin(2.0 * math.pi * x)
        x = x + amplitude * torch.stack([s[:, 1] * s[:, 2], s[:, 2] * s[:, 0], s[:, 0] * s[:, 1]], 1)
        x = x + inner * (jitter / n[0]) * noise
    return x, lambda local: number[flat(local)]


def _parts(case):
    if "cell" in case:
        return [(case["cell"], case["degree"], case["cells"], case.get("rule", ""))]
    return [("Hexahedron", 2, case["hexes"], "3x3x3"), ("Prism", 2, case["prisms"], "3x1x7"),
            ("Tetrahedron", 3, case["tets"], "4x3x2")]


def _mesh(case, seed):
    """The nodes [N][3] relative to the origin in the mesh's type, the origin, and per block
    (cell, degree, cells, rule, dofmap of a local lattice)."""
    xs, blocks, base = [], [], 0
    for i, (cell, p, cells, rule) in enumerate(_parts(case)):
        x, dofs = _box(cell, p, cells, seed + 7919 * i)
        x[:, 0] += 1.5 * i
        blocks.append((cell, p, cells, rule, lambda local, dofs=dofs, base=base: dofs(local) + base))
        xs.append(x)
        base += x.shape[0]
    x = torch.cat(xs)
    origin = 0.5 * (x.min(0).values + x.max(0).values)
    return (x - origin).to(torch.float32 if case.get("f32") else torch.float64), origin, blocks


def _geometry(case, seed):
    nodes, origin, blocks = _mesh(case, seed)
    gb = []
    for cell, p, _, _, dofs in blocks:
        local = np.rint(tg.refcell.lagrange_points(cell, p) * p).astype(np.int64)
        gb.append(tg.GeometryBlock(tg.CoordinateElement(cell, p), dofs(local).to(torch.int32).contiguous()))
    return tg.Geometry(gb, nodes, origin.tolist())


def _to_tiles(v):
    """Cell-major [cells][Q][LEN] to the tiled layout, padding lanes repeating the last cell."""
    c, q, n = v.shape
    pad = -c % TILE
    if pad:
        v = torch.cat([v, v[-1:].expand(pad, q, n)])
    return v.reshape(-1, TILE, q, n).permute(0, 2, 3, 1).reshape(-1)


def _from_tiles(flat, cells, q, n):
    return flat.reshape(-1, q, n, TILE).permute(0, 3, 1, 2).reshape(-1, q, n)[:cells]


def _cotangents(case, seed):
    """Per block, standard-normal cotangents of det J and K as flat tiled tensors."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 1)
    dt = torch.float64 if case["precision"] == "native" else torch.float32
    out = []
    for _, _, cells, rule in _parts(case):
        padded = -(-cells // TILE) * TILE
        out.append({name: torch.randn(padded * _rule_size(rule) * n, generator=gen, dtype=dt, device=DEV)
                    for name, n in (("detj", 1), ("pinv", 9))})
    return out


def _random_points(case, seed):
    """Reference points [cells][points][3] inside the cell, a little off its boundary."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 2)
    cell, shape = case["cell"], (case["cells"], case["points"], 3)
    u = torch.rand(shape, generator=gen, dtype=torch.float64, device=DEV)
    if cell == "Tetrahedron":
        u = torch.sort(u, dim=-1).values
        u = torch.diff(u, dim=-1, prepend=torch.zeros_like(u[..., :1]))
        centre = 0.25
    elif cell == "Prism":
        flip = u[..., 0] + u[..., 1] > 1.0
        u[..., :2] = torch.where(flip[..., None], 1.0 - u[..., :2], u[..., :2])
        centre = torch.tensor([1.0 / 3.0, 1.0 / 3.0, 0.5], dtype=torch.float64, device=DEV)
    else:
        centre = 0.5
    return centre + 0.9 * (u - centre)


# --------------------------------------------------------------------------------------------
# The calls.

def prepare(case, seed):
    kind = case["kind"]
    g = _geometry(case, seed)
    sets = [tg.PointSet(cell, *tg.refcell.collapsed_rule(cell, _counts(rule)))
            for cell, _, _, rule in _parts(case) if rule]
    if kind == "evaluate":
        s = {"kind": kind, "g": g, "pts": sets[0], "factors": FACTORS[case["factors"]], "precision": case["precision"],
             "sums": None}
        if case["measure"]:
            dt = torch.float32 if case["precision"] == "split" else g.dtype
            s["sums"] = torch.empty(case["cells"], dtype=dt, device=DEV)
        return s
    if kind == "batch":
        return {"kind": kind, "batch": tg.Batch(g, tg.QuadRule(sets), FACTORS["all"], precision=case["precision"])}
    if kind in ("vjp", "adjoint_batch"):
        ct = [{name: tg.QuadField([tg.geometry.QuadChunk(0, cells, flat)], cells, _rule_size(rule),
                                  LEN[name](3), TILE) for name, flat in c.items()}
              for c, (_, _, cells, rule) in zip(_cotangents(case, seed), _parts(case))]
        if kind == "vjp":
            tg.node_incidence(g, 0)
            return {"kind": kind, "g": g, "pts": sets[0], "ct": ct[0], "precision": case["precision"]}
        batch = tg.AdjointBatch(g, tg.QuadRule(sets), ct, precision=case["precision"], forward=FACTORS["all"])
        return {"kind": kind, "batch": batch, "precision": case["precision"]}
    # The points' images, in the mesh's type.
    xi = _random_points(case, seed)
    nodes, origin, blocks = _mesh(case, seed)
    x = _image(case, nodes, blocks[0], xi) + origin
    flat = _to_tiles(x).to(g.dtype)
    return {"kind": kind, "g": g, "precision": case["precision"], "tol": 1e-5 if case["f32"] else 1e-13,
            "x": tg.QuadField([tg.geometry.QuadChunk(0, case["cells"], flat)], case["cells"], case["points"], 3, TILE)}


def _flat(fields):
    return {name: f.chunks[0].data for name, f in fields.items()}


def _kept(grad, precision):
    """A single-precision adjoint's gradient, good to about seven digits, is kept in that type, as
    its cotangents are; the native one in 64 bits."""
    return grad if precision == "native" else grad.float()


def run(s):
    kind = s["kind"]
    if kind == "evaluate":
        out = _flat(tg.geometric_factors_block(s["g"], 0, s["pts"], s["factors"], precision=s["precision"],
                                               cell_measure=s["sums"]))
        if s["sums"] is not None:
            out["measure"] = tg.measure_block(s["g"], 0, s["pts"], sync=False, cell_sums=s["sums"])
            out["cell_measure"] = s["sums"]
        return out
    if kind == "batch":
        s["batch"].launch()
        return [_flat(f) for f in s["batch"].fields]
    if kind == "vjp":
        grad, fields = tg.vjp_block(s["g"], 0, s["pts"], s["ct"], precision=s["precision"], forward=FACTORS["all"])
        return {"grad": _kept(grad, s["precision"]), **_flat(fields)}
    if kind == "adjoint_batch":
        s["batch"].launch()
        return {"grad": _kept(s["batch"].grad, s["precision"]), "fields": [_flat(f) for f in s["batch"].fields]}
    # The step of a point's last iteration tells a program whether the point converged; its
    # value below the tolerance is rounding noise, so the comparison is the result.
    xi, step = tg.pull_back_block(s["g"], 0, s["x"], precision=s["precision"])
    return {"xi": xi.chunks[0].data, "converged": step.chunks[0].data <= s["tol"]}


# --------------------------------------------------------------------------------------------
# The same in 64 bits.

def _exponents(cell, p):
    return _lattice(cell, p)  # |a| <= p on simplices, a_d <= p per tensor direction


@functools.lru_cache(maxsize=None)
def _coefficients(cell, p):
    """C [m][k]: Lagrange function k (lattice order) = sum_m C[m][k] xi^m, by exact elimination."""
    nodes, ex = _lattice(cell, p), _exponents(cell, p)
    k = len(nodes)
    rows = []
    for i in range(k):
        x = [fractions.Fraction(int(v), p) for v in nodes[i]]
        rows.append([math.prod((x[d] ** int(e[d]) for d in range(len(x))), start=fractions.Fraction(1)) for e in ex]
                    + [fractions.Fraction(int(i == j)) for j in range(k)])
    for c in range(k):
        piv = next(r for r in range(c, k) if rows[r][c] != 0)
        rows[c], rows[piv] = rows[piv], rows[c]
        inv = 1 / rows[c][c]
        rows[c] = [v * inv if v else v for v in rows[c]]
        for r in range(k):
            f = rows[r][c]
            if r != c and f != 0:
                rows[r] = [a - f * b if b else a for a, b in zip(rows[r], rows[c])]
    return np.array([[float(v) for v in r[k:]] for r in rows])


def _monomials(cell, p, xi, derivative=None):
    """xi^a [..., m], or its derivative along one direction."""
    out = []
    for e in _exponents(cell, p):
        v = torch.ones_like(xi[..., 0])
        for d in range(xi.shape[-1]):
            n = int(e[d])
            if d == derivative:
                v = v * 0.0 if n == 0 else v * (n * xi[..., d] ** (n - 1))
            elif n:
                v = v * xi[..., d] ** n
        out.append(v)
    return torch.stack(out, -1)


def _image(case, nodes, block, xi):
    """X(xi) relative to the origin of points [cells][points][td] of their own in each cell."""
    cell, p, _, _, dofs = block
    y = nodes[dofs(_lattice(cell, p))].double()
    x0 = y[:, :1]
    coef = torch.einsum("mk,ckg->cmg", torch.from_numpy(_coefficients(cell, p)).to(DEV), y - x0)
    return torch.bmm(_monomials(cell, p, xi), coef) + x0


def _gauss_jacobi(m, a):
    """m-point Gauss rule on [0, 1] for the weight (1 - x)^a (Golub-Welsch, one Newton-polished
    symmetric eigenproblem), weights summing to 1 / (a + 1)."""
    n = np.arange(m, dtype=np.longdouble)
    s = 2 * n + a
    with np.errstate(divide="ignore", invalid="ignore"):
        diag = np.where(s == 0, 0.0, -(a * a) / (s * (s + 2)))
    if a == 0:
        diag[:] = 0
    k = np.arange(1, m, dtype=np.longdouble)
    s1 = 2 * k + a
    off = np.sqrt(4 * k * k * (k + a) * (k + a) / (s1 * s1 * (s1 + 1) * (s1 - 1)))
    jac = np.diag(diag) + np.diag(off, 1) + np.diag(off, -1)
    t, vecs = np.linalg.eigh(jac.astype(np.float64))
    t = t.astype(np.longdouble)
    for _ in range(2):  # Newton on the orthonormal recurrence's last polynomial
        q0, q1 = np.zeros(m, np.longdouble), np.ones(m, np.longdouble)
        d0, d1 = np.zeros(m, np.longdouble), np.zeros(m, np.longdouble)
        for i in range(m):
            b = off[i - 1] ** 2 if i else 0.0
            q0, q1, d0, d1 = q1, (t - diag[i]) * q1 - b * q0, d1, q1 + (t - diag[i]) * d1 - b * d0
        t = t - q1 / d1
    w = vecs[0] ** 2 / (a + 1)
    return (0.5 * (1 + t)).astype(np.float64), w


def _rule(cell, rule):
    """The collapsed Gauss-Jacobi product rule, first direction fastest."""
    alphas = {"Triangle": (0, 1), "Tetrahedron": (0, 1, 2), "Prism": (0, 1, 0), "Hexahedron": (0, 0, 0)}[cell]
    dirs = [_gauss_jacobi(m, a) for m, a in zip(_counts(rule), alphas)]
    grid = [g.ravel(order="F") for g in np.meshgrid(*[d[0] for d in dirs], indexing="ij")]
    w = math.prod(g.ravel(order="F") for g in np.meshgrid(*[d[1] for d in dirs], indexing="ij"))
    if cell == "Tetrahedron":
        grid = [grid[0] * (1 - grid[1]) * (1 - grid[2]), grid[1] * (1 - grid[2]), grid[2]]
    elif cell in ("Triangle", "Prism"):
        grid[0] = grid[0] * (1 - grid[1])
    return (torch.from_numpy(np.stack(grid, 1)).to(DEV), torch.from_numpy(np.ascontiguousarray(w)).to(DEV))


def _factors(x0, origin, coef, mono, names, td):
    """The named factors [c][q][LEN] of cells with monomial coefficients `coef` [c][m][3]."""
    out = {}
    if "points" in names:
        out["points"] = torch.matmul(mono[0], coef) + x0 + origin
    if set(names) <= {"points"}:
        return out
    cols = [torch.matmul(mono[1 + d], coef) for d in range(td)]  # J's columns [c][q][3]
    cross = torch.linalg.cross
    if td == 3:
        a, b, c = cols
        r = [cross(b, c), cross(c, a), cross(a, b)]
        det = (a * r[0]).sum(-1, keepdim=True)
        inv = [v / det for v in r]
    else:
        a, b = cols
        n = cross(a, b)
        n2 = (n * n).sum(-1, keepdim=True)
        det = torch.sqrt(n2)
        inv = [cross(b, n) / n2, cross(n, a) / n2]
        if "normals" in names:
            out["normals"] = n / det
    if "jacobian" in names:
        out["jacobian"] = torch.cat(cols, -1)
    if "detj" in names:
        out["detj"] = det
    if "pinv" in names:
        out["pinv"] = torch.stack(inv, -1).flatten(-2)
    return out


def _exact_block(nodes, origin, block, names, cts=None):
    """Factors of one block (cell-major, chunk by chunk); with cotangents also their gradient,
    added into nodes.grad."""
    cell, p, cells, rule, dofs = block
    td = TDIM[cell]
    pts, w = _rule(cell, rule)
    mono = [_monomials(cell, p, pts)] + [_monomials(cell, p, pts, d) for d in range(td)]
    dm = dofs(_lattice(cell, p))
    C = torch.from_numpy(_coefficients(cell, p)).to(DEV)
    step = max(TILE, 4_000_000 // len(pts) // TILE * TILE)
    parts = {n: [] for n in names}
    for c0 in range(0, cells, step):
        d = dm[c0: c0 + step]
        y = nodes[d].double()
        x0 = y[:, :1]
        coef = torch.einsum("mk,ckg->cmg", C, y - x0)
        f = _factors(x0, origin, coef, mono, names, td)
        if cts is not None:
            loss = 0.0
            for name, flat in cts.items():
                n = LEN[name](td)
                per = len(pts) * n
                loss = loss + (_from_tiles(flat[c0 * per: (c0 + (-(-d.shape[0] // TILE) * TILE)) * per], d.shape[0],
                                           len(pts), n).double() * f[name]).sum()
            loss.backward()
        for n in names:
            parts[n].append(f[n].detach())
        del f
    return {n: torch.cat(v) for n, v in parts.items()}, w


def exact(case, seed):
    kind = case["kind"]
    if kind == "pull_back":
        return {"xi": _to_tiles(_random_points(case, seed)), "converged": None}
    nodes, origin, blocks = _mesh(case, seed)
    if kind == "evaluate":
        names = FACTORS[case["factors"]]
        f, w = _exact_block(nodes, origin, blocks[0], names)
        out = {n: _to_tiles(f[n]) for n in names}
        if case["measure"]:
            sums = (f["detj"][..., 0] * w).sum(1)
            out["measure"], out["cell_measure"] = sums.sum().reshape(1), sums
        return out
    if kind == "batch":
        return [{n: _to_tiles(v) for n, v in _exact_block(nodes, origin, b, FACTORS["all"])[0].items()}
                for b in blocks]
    nodes.requires_grad_(True)
    fields = [{n: _to_tiles(v) for n, v in _exact_block(nodes, origin, b, FACTORS["all"], c)[0].items()}
              for b, c in zip(blocks, _cotangents(case, seed))]
    if kind == "vjp":
        return {"grad": nodes.grad, **fields[0]}
    return {"grad": nodes.grad, "fields": fields}


# --------------------------------------------------------------------------------------------
# What a pass cannot do without.

def work(case):
    """Bytes: dofmaps, every node once, the outputs (and cotangents) once. Operations: per point
    the sums over the monomials that X and the columns of J have, and det J and K; the adjoint
    about twice that; a pull-back five iterations a point."""
    es = 4 if case.get("f32") else 8
    out_es = 4 if case["precision"] == "split" else es
    nbytes = flops = 0.0
    for cell, p, cells, rule in _parts(case):
        td = TDIM[cell]
        ex = _exponents(cell, p)
        k = len(ex)
        per_cell = {"Triangle": p * p / 2, "Tetrahedron": p ** 3 / 6, "Prism": p ** 3 / 2, "Hexahedron": p ** 3}[cell]
        nbytes += cells * (4 * k + per_cell * 3 * es)
        terms = k - 1 + sum(int((ex[:, d] > 0).sum()) for d in range(td))
        point = 6 * terms + (55 if td == 3 else 40)
        if case["kind"] == "pull_back":
            nbytes += cells * case["points"] * 7 * es
            flops += cells * case["points"] * 5 * (point + 18)
            continue
        nq = _rule_size(rule)
        names = FACTORS[case.get("factors", "all")]
        nbytes += cells * nq * sum(LEN[n](td) for n in names) * out_es
        flops += cells * nq * point
        if case.get("measure"):
            nbytes += cells * out_es
        if case["kind"] in ("vjp", "adjoint_batch"):
            nbytes += cells * nq * 10 * (8 if case["precision"] == "native" else 4) + cells * per_cell * 24
            flops += cells * nq * (point + 90)
    return {"bytes": nbytes, "flops": flops}
