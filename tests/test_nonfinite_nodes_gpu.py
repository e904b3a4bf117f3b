"""A node coordinate that is not finite makes its cells' points, Jacobians, det J and K so at every point of
the rule, the middle point of an odd Gauss rule (where the node's function is zero) included, as the sums of
the loops kernel do. Other cells are not disturbed."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("local", [0, 3, -1])
@pytest.mark.parametrize("cell,precision", [("Hexahedron", "native"), ("Hexahedron", "df64"), ("Hexahedron", "split"),
                                            ("Hexahedron", "f32"), ("Prism", "native"), ("Prism", "df64"),
                                            ("Quadrilateral", "native")])
def test_every_point_of_the_cell(cuda, cell, precision, local, value):
    td = tg.refcell.tdim(cell)
    mesh = meshes.square_box(cell, 4, 2) if td == 2 else meshes.curved_box(cell, 3, 2, jitter=0.01)
    cells = mesh.blocks[0].cells
    node = cells[3, local]
    hit = (cells == node).any(axis=1)
    pts, _ = tg.refcell.collapsed_rule(cell, (3, 3, 3)[:td])
    ps = tg.PointSet(cell, pts, np.ones(len(pts)))
    names = ("points", "jacobian", "detj", "pinv")
    dtype = torch.float32 if precision == "f32" else torch.float64
    mode = "native" if precision == "f32" else precision
    g = tg.Geometry.from_host(mesh, dtype=dtype)
    want = tg.geometric_factors_block(g, 0, ps, names, precision=mode)
    g.nodes[int(node)] = value
    got = tg.geometric_factors_block(g, 0, ps, names, precision=mode)
    for f in names:
        a, w = got[f].to_host_cell_major(), want[f].to_host_cell_major()
        if f in ("points", "detj", "pinv"):
            assert not np.isfinite(a[hit]).any(), f
        assert np.array_equal(a[~hit], w[~hit]), f
