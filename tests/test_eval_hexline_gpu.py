"""The FP32 line kernel of hexahedra (f32 meshes and split precision) against the oracle at the point sets,
ranges and tiles where its indexing can go wrong, with the f32 tolerance of the parity tests (1e-5 scaled by
the element's amplification, the origin ratio and, for K, the condition number), and the FP64 recompute of
near-degenerate cells."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

FACTORS = ("points", "jacobian", "detj", "pinv")
KEYS = {"points": "x", "jacobian": "j", "detj": "detj", "pinv": "k"}


def rule_of(kind):
    rng = np.random.default_rng(3)
    if kind == "one":
        return np.full((1, 3), 0.5)
    if kind == "scattered":
        return rng.uniform(0.05, 0.95, size=(7, 3))
    counts = {"rule": (3, 3, 3), "long": (6, 2, 2), "planes": (2, 1, 13), "wide": (9, 9, 2), "large": (9, 9, 9)}[kind]
    pts, _ = tg.refcell.collapsed_rule("Hexahedron", counts)
    return pts[rng.permutation(len(pts))] if kind == "planes" else pts


def check(mesh, degree, pts, precision, **kw):
    g = tg.Geometry.from_host(mesh, dtype=torch.float32 if precision == "native" else torch.float64)
    ps = tg.PointSet("Hexahedron", pts, np.ones(len(pts)))
    got = tg.geometric_factors_block(g, 0, ps, FACTORS, precision=precision, **kw)
    absx = g.nodes.double().cpu().numpy() + np.array(g.origin[:3])
    want = orc.eval_block("Hexahedron", degree, absx, mesh.blocks[0].cells, pts, factors=[KEYS[f] for f in FACTORS])
    s = orc.tolerance_scale("Hexahedron", degree, "Equispaced", pts) * orc.node_ratio("Hexahedron", degree)
    if precision == "native":
        s *= orc.origin_ratio(absx, np.array(g.origin[:3]), want["j"])
    cond = orc.condition_scale(want["j"], 3, 3)
    for f in FACTORS:
        err = orc.rel_err(got[f].to_host_cell_major(), want[KEYS[f]])
        assert err < orc.TOL_F32 * s * (cond if f == "pinv" else 1.0), (f, err)
    return g, ps, got


@pytest.mark.parametrize("precision", ["native", "split"])
@pytest.mark.parametrize("kind", ["one", "scattered", "rule", "long", "planes", "wide", "large"])
@pytest.mark.parametrize("degree", [1, 2])
def test_point_sets(cuda, degree, kind, precision):
    mesh = meshes.curved_box("Hexahedron", 3, degree, jitter=0.02).first_cells(21)
    g, ps, got = check(mesh, degree, rule_of(kind), precision)
    for f in FACTORS:  # one factor at a time, and in chunks: the same values
        one = tg.geometric_factors_block(g, 0, ps, (f,), precision=precision)[f]
        assert torch.equal(got[f].chunks[0].data, one.chunks[0].data), f
    parts = tg.geometric_factors_block(g, 0, ps, FACTORS, precision=precision, max_chunk_cells=16)
    for f in FACTORS:
        assert np.array_equal(got[f].to_host_cell_major(), parts[f].to_host_cell_major()), f


@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("tile", [1, 2, 8])
def test_tiles_of_f32(cuda, tile, degree):
    mesh = meshes.curved_box("Hexahedron", 3, degree, jitter=0.02).first_cells(21)
    g, ps, got = check(mesh, degree, rule_of("rule"), "native")
    other = tg.geometric_factors_block(g, 0, ps, FACTORS, tile=tile)
    for f in FACTORS:
        assert np.array_equal(got[f].to_host_cell_major(), other[f].to_host_cell_major()), f


def test_near_degenerate_cells_are_recomputed(cuda):
    """Cells flattened by 1e-5 exceed the condition limit of 256: det J and K come from FP64 and are counted,
    all of their points and no other."""
    mesh = meshes.cube_box("Hexahedron", 4, 2)
    pts = rule_of("rule")
    flat = mesh.nodes.copy()
    flat[:, 2] *= 1e-5
    mesh = meshes.combine([mesh, meshes.HostMesh(3, flat, mesh.blocks)], [(0, 0, 0), (2, 0, 0)])
    cells = np.concatenate([b.cells for b in mesh.blocks])
    mesh = meshes.HostMesh(3, mesh.nodes, [meshes.HostBlock("Hexahedron", 2, cells)])
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    ps = tg.PointSet("Hexahedron", pts, np.ones(len(pts)))
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    got = tg.geometric_factors_block(g, 0, ps, ("detj", "pinv"), precision="split", recomputed=count)
    assert int(count.item()) == 64 * len(pts)
    want = tg.geometric_factors_block(g, 0, ps, ("detj", "pinv"))
    for f in ("detj", "pinv"):
        a, b = got[f].to_host_cell_major()[64:], want[f].to_host_cell_major()[64:]
        assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max(), f
