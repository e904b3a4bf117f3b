"""A cotangent that is not finite at a rule's middle point, where the functions of a tensor cell's outer nodes and
their derivatives are zero: every node of the cell gets NaN, as through the Lagrange functions (0 times NaN),
and the nodes of no other cell."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("factor", ["points", "detj", "pinv"])
@pytest.mark.parametrize("cell", ["Hexahedron", "Quadrilateral"])
def test_middle_point(cuda, cell, factor, value):
    td = tg.refcell.tdim(cell)
    mesh = meshes.square_box(cell, 5, 2) if td == 2 else meshes.curved_box(cell, 3, 2, jitter=0.01)
    nc = mesh.blocks[0].num_cells
    pts, w = tg.refcell.collapsed_rule(cell, (3, 3, 3)[:td])
    middle = int(np.flatnonzero((np.abs(pts - 0.5) < 1e-12).all(axis=1))[0])
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    ln = {"points": td, "detj": 1, "pinv": td * td}[factor]
    ct = tg.QuadField.uninit(nc, len(pts), ln, 16, torch.float64)
    v = np.random.default_rng(2).standard_normal((nc + -nc % 16, len(pts), ln))
    v[nc:] = 0.0
    v[7, middle] = value
    ct.chunks[0].data.copy_(torch.from_numpy(v.reshape(-1, 16, len(pts), ln).transpose(0, 2, 3, 1).ravel().copy()))
    grad = tg.vjp_block(g, 0, tg.PointSet(cell, pts, w), {factor: ct})[0].cpu().numpy()
    hit = np.zeros(len(grad), dtype=bool)
    hit[mesh.blocks[0].cells[7]] = True
    assert not np.isfinite(grad[hit]).any()
    assert np.isfinite(grad[~hit]).all()
