"""The f64 polynomial adjoint against the oracle's restated adjoint (which a CPU test checks against
central differences) at the point sets and sizes where its stages can go wrong: one point, points
that share no line, more planes and lines than a CTA holds at a time, permuted rules, missing
cotangents, ragged cell counts, meshes of few and of many CTAs. Tolerance as the adjoint tests':
1e-11 of the largest node cotangent."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

CELLS = [("Tetrahedron", 1), ("Tetrahedron", 2), ("Tetrahedron", 3), ("Hexahedron", 1), ("Hexahedron", 2),
         ("Prism", 1), ("Prism", 2), ("Triangle", 1), ("Triangle", 3), ("Quadrilateral", 1), ("Quadrilateral", 2)]


def mesh_of(cell, degree, n):
    if cell in ("Triangle", "Quadrilateral"):
        m = meshes.square_box(cell, n, degree)
        m.nodes = meshes.jitter_interior(m.nodes, m.nodes, 0.03 / n, 2026)
        return m
    return meshes.curved_box(cell, n, degree, jitter=0.01)


def rule_of(cell, kind):
    td = tg.refcell.tdim(cell)
    rng = np.random.default_rng(td)
    if kind == "one":
        return np.full((1, td), 0.2)
    if kind == "scattered":
        return rng.uniform(0.05, 0.3, size=(9, td))
    counts = {"rule": (3, 3, 3), "planes": (2, 1, 11), "lines": (2, 14, 2), "large": (9, 9, 10)}[kind][:td]
    pts, _ = tg.refcell.collapsed_rule(cell, counts)
    return pts[rng.permutation(len(pts))] if kind in ("planes", "lines") else pts


def run(mesh, cell, degree, pts, factors):
    td = tg.refcell.tdim(cell)
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    ps = tg.PointSet(cell, pts, np.ones(len(pts)))
    nc, nq = mesh.blocks[0].num_cells, len(pts)
    rng = np.random.default_rng(7)
    host = {"points": np.zeros((nc, nq, td)), "detj": np.zeros((nc, nq)), "pinv": np.zeros((nc, nq, td * td))}
    ct = {}
    for f in factors:
        host[f] = rng.standard_normal(host[f].shape)
        ln = {"points": td, "detj": 1, "pinv": td * td}[f]
        q = tg.QuadField.uninit(nc, nq, ln, 16, torch.float64)
        v = np.concatenate([host[f].reshape(nc, nq, ln), np.zeros((-nc % 16, nq, ln))])
        q.chunks[0].data.copy_(torch.from_numpy(v.reshape(-1, 16, nq, ln).transpose(0, 2, 3, 1).ravel().copy()))
        ct[f] = q
    names = ("points", "jacobian", "detj", "pinv")
    grad, fused = tg.vjp_block(g, 0, ps, ct, forward=names)
    alone, _ = tg.vjp_block(g, 0, ps, ct)
    assert torch.equal(grad, alone)
    plain = tg.geometric_factors_block(g, 0, ps, names)
    for k in names:  # the same stages: the same bits
        assert torch.equal(fused[k].chunks[0].data, plain[k].chunks[0].data), k
    absx = g.nodes.cpu().numpy() + np.array(g.origin[: g.gdim])
    want = orc.vjp(cell, degree, absx, mesh.blocks[0].cells, pts, host["points"], host["detj"], host["pinv"])
    assert orc.rel_err(grad.cpu().numpy(), want) < 1e-11


@pytest.mark.parametrize("kind", ["one", "scattered", "rule", "planes", "lines", "large"])
@pytest.mark.parametrize("cell,degree", CELLS)
def test_point_sets(cuda, cell, degree, kind):
    run(mesh_of(cell, degree, 5 if cell in ("Triangle", "Quadrilateral") else 2).first_cells(21), cell, degree,
        rule_of(cell, kind), ("points", "detj", "pinv"))


@pytest.mark.parametrize("factors", [("points",), ("detj",), ("pinv",)])
@pytest.mark.parametrize("cell,degree", [("Hexahedron", 2), ("Tetrahedron", 2), ("Quadrilateral", 2)])
def test_missing_cotangents(cuda, cell, degree, factors):
    run(mesh_of(cell, degree, 4), cell, degree, rule_of(cell, "rule"), factors)


@pytest.mark.parametrize("cell,n,cells,kind", [("Hexahedron", 22, 10001, "rule"), ("Prism", 18, 9999, "planes"),
                                               ("Quadrilateral", 105, 10930, "lines")])
def test_wide_groups(cuda, cell, n, cells, kind):
    """Meshes large enough for 32-cell CTAs, the last one ragged."""
    run(mesh_of(cell, 2, n).first_cells(cells), cell, 2, rule_of(cell, kind), ("points", "detj", "pinv"))
