"""The f64 polynomial evaluation (line by line of the point set) against the oracle at the sizes
and point sets where its indexing can go wrong: one point, points that share no line, lines longer
than a part, permuted rules, rules beyond the staged size, more planes than a batch, facet rules,
flags, ragged cell counts, tiles and chunks. Tolerances are the f64 ones of the parity tests (the
reference's 1e-12 scaled by the element's amplification, origin and condition ratios)."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

KEYS = {"points": "x", "jacobian": "j", "detj": "detj", "pinv": "k", "normals": "normals",
        "facet_normals": "facet_normals"}
CELLS = [("Tetrahedron", 1, 3), ("Tetrahedron", 2, 3), ("Tetrahedron", 3, 3), ("Hexahedron", 1, 3),
         ("Hexahedron", 2, 3), ("Prism", 1, 3), ("Prism", 2, 3), ("Triangle", 1, 2), ("Triangle", 2, 3),
         ("Triangle", 3, 2), ("Triangle", 3, 3), ("Quadrilateral", 1, 3), ("Quadrilateral", 2, 2),
         ("Quadrilateral", 2, 3)]


def mesh_of(cell, degree, gd):
    if cell in ("Triangle", "Quadrilateral"):
        m = meshes.square_box(cell, 5, degree)
        m.nodes = meshes.jitter_interior(m.nodes, m.nodes, 0.005, 2026)
        if gd == 3:
            m = meshes.HostMesh(3, np.concatenate([m.nodes, 0.1 * np.sin(3.0 * m.nodes[:, :1])], 1), m.blocks)
        return m.first_cells(23)
    return meshes.curved_box(cell, 3 if cell == "Hexahedron" else 2, degree, jitter=0.01).first_cells(23)


def rule_of(cell, kind):
    td = tg.refcell.tdim(cell)
    rng = np.random.default_rng(td)
    if kind == "one":
        return np.full((1, td), 0.2)
    if kind == "scattered":
        return rng.uniform(0.05, 0.3, size=(7, td))
    counts = {"long": (6, 2, 2), "planes": (2, 1, 11), "large": (10, 10, 10)}[kind][:td]
    pts, _ = tg.refcell.collapsed_rule(cell, counts)
    return pts[rng.permutation(len(pts))] if kind == "planes" else pts


def check(mesh, g, cell, degree, pts, got, names, td, ref_normals=None, flags=None):
    absx = g.nodes.cpu().numpy() + np.array(g.origin[: g.gdim])
    want = orc.eval_block(cell, degree, absx, mesh.blocks[0].cells, pts, factors=["j"] + [KEYS[f] for f in names],
                          ref_normals=ref_normals, flags=flags)
    s = orc.tolerance_scale(cell, degree, "Equispaced", pts) * orc.node_ratio(cell, degree)
    s *= orc.origin_ratio(absx, np.array(g.origin[: g.gdim]), want["j"])
    cond = orc.condition_scale(want["j"], td, g.gdim)
    for f in names:
        err = orc.rel_err(got[f].to_host_cell_major(), want[KEYS[f]])
        assert err < orc.TOL_F64 * s * (cond if f in ("pinv", "normals", "facet_normals") else 1.0), (f, err)


@pytest.mark.parametrize("kind", ["one", "scattered", "long", "planes", "large"])
@pytest.mark.parametrize("cell,degree,gd", CELLS)
def test_point_sets(cuda, cell, degree, gd, kind):
    mesh = mesh_of(cell, degree, gd)
    td = tg.refcell.tdim(cell)
    flags = (np.arange(mesh.blocks[0].num_cells) % 3 == 0).astype(np.uint32)
    g = tg.Geometry.from_host(mesh, dtype=torch.float64, flags=[flags])
    pts = rule_of(cell, kind)
    ps = tg.PointSet(cell, pts, np.ones(len(pts)))
    names = ("points", "jacobian", "detj", "pinv") + (("normals",) if td + 1 == gd else ())
    got = tg.geometric_factors_block(g, 0, ps, names)
    check(mesh, g, cell, degree, pts, got, names, td, flags=flags if td < gd else None)
    # One output tile or another, several chunks, and one factor at a time: the same values.
    for kw in ({"tile": 1}, {"tile": 4, "max_chunk_cells": 8}):
        other = tg.geometric_factors_block(g, 0, ps, names, **kw)
        for f in names:
            assert np.array_equal(got[f].to_host_cell_major(), other[f].to_host_cell_major()), f
    for f in names:
        one = tg.geometric_factors_block(g, 0, ps, (f,))[f]
        assert torch.equal(got[f].chunks[0].data, one.chunks[0].data), f


@pytest.mark.parametrize("cell,degree", [("Tetrahedron", 2), ("Hexahedron", 2), ("Prism", 2), ("Hexahedron", 1)])
def test_facet_rules(cuda, cell, degree):
    mesh = mesh_of(cell, degree, 3)
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    ps = tg.facet_point_set(cell, 3)
    names = ("points", "detj", "facet_normals")
    got = tg.geometric_factors_block(g, 0, ps, names)
    check(mesh, g, cell, degree, ps.points, got, names, 3, ref_normals=ps.ref_normals)


def test_clamped_nodes_and_padding(cuda):
    """A node index past the last node reads the last node; padding lanes repeat the last cell."""
    mesh = mesh_of("Tetrahedron", 2, 3)
    bad = mesh.blocks[0].cells.copy()
    bad[5, 3] = 10 ** 6
    clamped = bad.copy()
    clamped[5, 3] = mesh.num_nodes - 1
    pts, w = tg.refcell.gauss_rule("Tetrahedron", 4)
    ps = tg.PointSet("Tetrahedron", pts, w)
    out = []
    for cells in (bad, clamped):
        m = meshes.HostMesh(3, mesh.nodes, [meshes.HostBlock("Tetrahedron", 2, cells)])
        out.append(tg.jacobians_block(tg.Geometry.from_host(m), 0, ps).chunks[0].data)
    assert torch.equal(out[0], out[1])
    v = out[0].reshape(2, -1, 16)[1]
    assert torch.equal(v[:, 7:], v[:, 6:7].expand(-1, 9))
