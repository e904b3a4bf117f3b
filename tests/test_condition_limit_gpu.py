"""Split precision's condition limit at infinity: no point with a finite J and K is recomputed, also where
the squares of the estimate overflow f32."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,degree", [("Hexahedron", 1), ("Hexahedron", 2), ("Tetrahedron", 2)])
def test_infinite_limit(cuda, cell, degree):
    mesh = meshes.cube_box(cell, 3, degree)
    mesh.nodes = mesh.nodes * np.array([1.0, 1.0, 2.0 ** -90])  # |K| near 2^92: its square passes f32
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    pts, w = tg.refcell.collapsed_rule(cell, (2, 2, 2))
    ps = tg.PointSet(cell, pts, w)
    for limit, expected in ((float("inf"), 0), (1e30, mesh.blocks[0].num_cells * len(pts))):
        count = torch.zeros(1, dtype=torch.int64, device="cuda")
        got = tg.geometric_factors_block(g, 0, ps, ("detj", "pinv"), precision="split", cond_limit=limit,
                                         recomputed=count)
        assert int(count.item()) == expected
        assert torch.isfinite(got["pinv"].chunks[0].data).all()
