"""The rows kernel's runs of whole tiles (more tiles than SMs, where equal runs would start too many tiles):
the same bits as equal runs of fewer cells, in split precision also with the queue of ill-conditioned points."""

import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu

FACTORS = ("points", "jacobian", "detj", "pinv")


@pytest.mark.parametrize("precision", ["f32", "split"])
@pytest.mark.parametrize("tiles", [229, 290, 304])  # of 16 chunks, on 152 SMs: 115, 145 and 152 runs of two
def test_whole_tiles_equal_equal_runs(cuda, tiles, precision):
    mesh = meshes.curved_box("Tetrahedron", 19, 4, jitter=0.01).first_cells(128 * tiles - 5)
    g = tg.Geometry.from_host(mesh, dtype=torch.float32 if precision == "f32" else torch.float64)
    ps = tg.PointSet("Tetrahedron", *tg.refcell.collapsed_rule("Tetrahedron", (5, 5, 5)))
    kw = {"precision": "native"} if precision == "f32" else {"precision": "split", "cond_limit": 12.0}
    one = tg.geometric_factors_block(g, 0, ps, FACTORS, **kw)
    parts = tg.geometric_factors_block(g, 0, ps, FACTORS, max_chunk_cells=128 * 76, **kw)
    for f in FACTORS:
        assert torch.equal(one[f].chunks[0].data, torch.cat([c.data for c in parts[f].chunks])), f
