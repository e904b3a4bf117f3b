"""Collapsed cells in double-float precision, on the kernels that assemble their values with df_to_f64
(surfaces, planar cells, pyramids, volume cells with facet normals): 0 / 0 is not
finite, and the other cells are not disturbed."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu


def mesh_of(cell, degree, gd):
    if cell == "Pyramid":
        return meshes.hex_prism_pyramid_box(2, degree)
    if cell in ("Triangle", "Quadrilateral"):
        m = meshes.square_box(cell, 4, degree)
        return m if gd == 2 else meshes.HostMesh(3, np.concatenate([m.nodes, m.nodes[:, :1] ** 2], 1), m.blocks)
    return meshes.curved_box(cell, 2, degree, jitter=0.01)


@pytest.mark.parametrize("cell,degree,gd", [("Triangle", 1, 3), ("Triangle", 4, 3), ("Triangle", 2, 2),
                                            ("Quadrilateral", 2, 3), ("Quadrilateral", 1, 2), ("Pyramid", 1, 3),
                                            ("Hexahedron", 2, 3), ("Prism", 1, 3), ("Tetrahedron", 2, 3)])
def test_collapsed_cell(cuda, cell, degree, gd):
    mesh = mesh_of(cell, degree, gd)
    b = next(i for i, blk in enumerate(mesh.blocks) if blk.cell == cell)
    cells = mesh.blocks[b].cells.copy()
    cells[2] = cells[2, 0]
    mesh = meshes.HostMesh(gd, mesh.nodes, [meshes.HostBlock(cell, degree, cells)])
    td = tg.refcell.tdim(cell)
    pts, _ = tg.refcell.collapsed_rule(cell, (3, 2, 2)[:td])
    ref = np.tile(np.eye(td)[0], (len(pts), 1))
    names = ("detj", "pinv", "normals" if td < gd else "facet_normals")
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    ps = tg.PointSet(cell, pts, np.ones(len(pts)), ref_normals=ref if td == gd else None)
    got = tg.geometric_factors_block(g, 0, ps, names, precision="df64")
    with tg.with_strategy("loops"):
        want = tg.geometric_factors_block(g, 0, ps, names)
    keep = np.arange(len(cells)) != 2
    for f in names:
        a, w = got[f].to_host_cell_major(), want[f].to_host_cell_major()
        assert np.abs(a[keep] - w[keep]).max() <= 3e-13 * np.abs(w[keep]).max(), f
    # The shifted nodes of the collapsed cell are zeros, and so are J and det J: K and the normals are 0 / 0.
    assert np.all(got["detj"].to_host_cell_major()[2] == 0.0)
    for f in names[1:]:
        assert not np.isfinite(got[f].to_host_cell_major()[2]).any(), f
