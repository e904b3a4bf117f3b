"""The tcgen05 kernel with one accumulator row per cell (volume cells of 28 to 56 nodes, 64 on f32
meshes): against the oracle at the f32 tolerance around the sizes where it can go wrong (one cell, a
tile of 128 cells more or less, a chunk of 8 points more or less, node counts that fill their
k-steps or not), and the equal runs of its work against whole tiles per CTA (GPU)."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

FACTORS = ("points", "jacobian", "detj", "pinv")
KEYS = {"points": "x", "jacobian": "j", "detj": "detj", "pinv": "k"}


def evaluate(mesh, cell, pts, precision, **kw):
    g = tg.Geometry.from_host(mesh, dtype=torch.float32 if precision == "f32" else torch.float64)
    ps = tg.PointSet(cell, pts, np.ones(len(pts)))
    with tg.with_strategy("tensor"):
        got = tg.geometric_factors_block(g, 0, ps, FACTORS, precision="split" if precision == "split" else "native", **kw)
        assert tg.last_kernel_family() == "tensor"
    return g, got


@pytest.mark.parametrize("precision", ["f32", "split"])
@pytest.mark.parametrize("cell,degree,n,cells,points", [
    ("Pyramid", 3, 3, 129, 9),       # 30 nodes of 32
    ("Tetrahedron", 4, 3, 1, 1),     # 35 nodes of 40
    ("Tetrahedron", 4, 3, 127, 7),
    ("Prism", 3, 5, 128, 8),         # 40 nodes, all of its k-steps
    ("Tetrahedron", 5, 4, 257, 17),  # 56 nodes, all of its k-steps
    ("Hexahedron", 3, 6, 130, 10),   # 64 nodes
    ("Tetrahedron", 4, 15, 19600, 9),
])
def test_edges_match_the_oracle(cuda, cell, degree, n, cells, points, precision):
    mesh = meshes.curved_box(cell, n, degree, jitter=0.02)
    mesh.blocks[0].cells = mesh.blocks[0].cells[:cells]
    pts, _ = tg.refcell.gauss_rule(cell, 8)
    pts = pts[np.random.default_rng(3).permutation(len(pts))][:points]
    g, got = evaluate(mesh, cell, pts, precision)
    absx = g.nodes.double().cpu().numpy() + np.array(g.origin[:3])
    want = orc.eval_block(cell, degree, absx, mesh.blocks[0].cells, pts, factors=[KEYS[f] for f in FACTORS])
    nodes = orc.node_ratio(cell, degree)
    s_val = orc.tolerance_scale(cell, degree, "Equispaced", pts, "values") * nodes
    s_der = orc.tolerance_scale(cell, degree, "Equispaced", pts) * nodes
    if precision == "f32":
        r = orc.origin_ratio(absx, np.array(g.origin[:3]), want["j"])
        s_val, s_der = s_val * r, s_der * r
    scale = {"points": s_val, "jacobian": s_der, "detj": s_der,
             "pinv": s_der * orc.condition_scale(want["j"], 3, 3)}
    for f in FACTORS:
        err = orc.rel_err(got[f].to_host_cell_major(), want[KEYS[f]])
        assert err < orc.TOL_F32 * scale[f], (f, err)


@pytest.mark.parametrize("precision", ["f32", "split"])
def test_runs_across_tiles_equal_whole_tiles(cuda, precision):
    """154 tiles of 27 chunks go in equal runs that cross tiles, 38 of them in parts of a tile: the
    same bits; in split precision also with the queue of ill-conditioned points in use."""
    mesh = meshes.curved_box("Tetrahedron", 15, 5, jitter=0.02)
    mesh.blocks[0].cells = mesh.blocks[0].cells[:19600]
    pts, _ = tg.refcell.gauss_rule("Tetrahedron", 10)
    kw = {"cond_limit": 12.0} if precision == "split" else {}
    one = evaluate(mesh, "Tetrahedron", pts, precision, **kw)[1]
    parts = evaluate(mesh, "Tetrahedron", pts, precision, max_chunk_cells=4864, **kw)[1]
    for f in FACTORS:
        rows = torch.cat([c.data for c in parts[f].chunks])
        assert torch.equal(one[f].chunks[0].data, rows), f
