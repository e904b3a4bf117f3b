"""The f64 adjoint at one point (two on P3 tetrahedra) of blocks that fill the device, which the node-row kernel
runs: against the oracle's adjoint (1e-11 of the largest node cotangent, the adjoint tests' bound), and its
forward fields against the evaluation's (1e-12 of the largest value)."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("factors", [("points", "detj", "pinv"), ("detj",)])
@pytest.mark.parametrize("cell,n,degree,npts", [("Tetrahedron", 12, 2, 1), ("Tetrahedron", 12, 3, 2),
                                                ("Hexahedron", 22, 2, 1), ("Prism", 17, 2, 1), ("Triangle", 70, 2, 1)])
def test_few_points(cuda, cell, n, degree, npts, factors):
    if cell == "Triangle":
        mesh = meshes.square_box(cell, n, degree)
        mesh.nodes = meshes.jitter_interior(mesh.nodes, mesh.nodes, 0.03 / n, 2026)
    else:
        mesh = meshes.curved_box(cell, n, degree, jitter=0.05 / n)
    nc, td = mesh.blocks[0].num_cells, tg.refcell.tdim(cell)
    assert nc >= 64 * 152
    rng = np.random.default_rng(1)
    pts = rng.uniform(0.1, 0.3, size=(npts, td))
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    ps = tg.PointSet(cell, pts, np.ones(npts))
    host, ct = {}, {}
    for f, ln in (("points", td), ("detj", 1), ("pinv", td * td)):
        host[f] = rng.standard_normal((nc, npts, ln)) if f in factors else np.zeros((nc, npts, ln))
        if f in factors:
            ct[f] = tg.QuadField.uninit(nc, npts, ln, 16, torch.float64)
            v = np.concatenate([host[f], np.zeros((-nc % 16, npts, ln))])
            ct[f].chunks[0].data.copy_(torch.from_numpy(v.reshape(-1, 16, npts, ln).transpose(0, 2, 3, 1).ravel().copy()))
    names = ("points", "jacobian", "detj", "pinv")
    grad, fused = tg.vjp_block(g, 0, ps, ct, forward=names)
    plain = tg.geometric_factors_block(g, 0, ps, names)
    for k in names:
        a, b = fused[k].to_host_cell_major(), plain[k].to_host_cell_major()
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), k
    absx = g.nodes.cpu().numpy() + np.array(g.origin[: g.gdim])
    want = orc.vjp(cell, degree, absx, mesh.blocks[0].cells, pts, host["points"], host["detj"].reshape(nc, npts),
                   host["pinv"])
    assert orc.rel_err(grad.cpu().numpy(), want) < 1e-11
