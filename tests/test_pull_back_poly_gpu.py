"""The polynomial pull-back kernels (simplices, tensor cells and prisms of degree 1-3): single
iterates and converged points against the oracle, at ragged cell counts, tiles, point counts and
chunks. The oracle forms X and J from Lagrange products; per iterate the two differ by the rounding
of X (a few eps of coordinates of size 1) times |K| <= 10 on these meshes, about 1e-14, amplified by
at most the maps' second derivatives over three iterates: 1e-11 leaves two orders."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def mesh_of(cell, degree, gd):
    if cell == "Triangle" and gd == 3:
        return meshes.perturbed_radius(meshes.sphere(1, degree), 0.02)
    if cell in ("Triangle", "Quadrilateral"):
        m = meshes.square_box(cell, 3, degree)
        m.nodes = meshes.jitter_interior(m.nodes, m.nodes, 0.01, 2026)
        if gd == 3:
            m = meshes.HostMesh(3, np.concatenate([m.nodes, 0.1 * np.sin(3.0 * m.nodes[:, :1])], 1), m.blocks)
        return m
    return meshes.curved_box(cell, 2, degree, jitter=0.01)


CASES = [("Tetrahedron", 1, 3), ("Tetrahedron", 2, 3), ("Tetrahedron", 3, 3), ("Hexahedron", 1, 3),
         ("Hexahedron", 2, 3), ("Hexahedron", 3, 3), ("Prism", 1, 3), ("Prism", 2, 3), ("Prism", 3, 3),
         ("Triangle", 1, 2), ("Triangle", 3, 2), ("Triangle", 2, 3), ("Quadrilateral", 1, 3), ("Quadrilateral", 2, 2),
         ("Quadrilateral", 3, 3)]


@pytest.mark.parametrize("tile,nq,chunk", [(16, 1, None), (1, 5, None), (4, 13, 20)])
@pytest.mark.parametrize("cell,degree,gd", CASES)
def test_poly_pull_back(cuda, cell, degree, gd, tile, nq, chunk):
    mesh = mesh_of(cell, degree, gd).first_cells(29)  # one full 16-cell group and a ragged one
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    cells = mesh.blocks[0].cells
    td = tg.refcell.tdim(cell)
    rng = np.random.default_rng(degree + 10 * td)
    ref = rng.uniform(0.05, 0.3, size=(nq, td))
    absx = g.nodes.cpu().numpy() + np.array(g.origin[:gd])
    x = orc.eval_block(cell, degree, absx, cells, ref, factors=("x",))["x"]
    field = tg.QuadField.uninit(len(cells), nq, gd, tile, torch.float64, max_chunk_cells=chunk)
    for ch in field.chunks:
        v = x[ch.first_cell: ch.first_cell + ch.num_cells]
        v = np.concatenate([v, np.repeat(v[-1:], -len(v) % tile, axis=0)])
        ch.data.copy_(torch.from_numpy(v.reshape(-1, tile, nq, gd).transpose(0, 2, 3, 1).ravel().copy()))
    for its in (1, 3, 16):
        xi, step = tg.pull_back_block(g, 0, field, max_iterations=its)
        want_xi, want_step = orc.pull_back(cell, degree, absx, cells, x, max_iterations=its)
        assert np.abs(xi.to_host_cell_major() - want_xi).max() < 1e-11
        assert np.abs(step.to_host_cell_major()[..., 0] - want_step).max() < 1e-11
    assert np.abs(xi.to_host_cell_major() - ref[None]).max() < 1e-11
    split, sstep = tg.pull_back_block(g, 0, field, precision="split")
    assert np.abs(split.to_host_cell_major() - ref[None]).max() < 1e-11
    assert sstep.to_host_cell_major().max() <= 1e-13
    # An f32 mesh: rounding of X and x to 2^-24 times |K| <= 10 and the sums' few terms: 1e-5.
    g32 = tg.Geometry(g.blocks, g.nodes.float(), g.origin)
    f32 = tg.QuadField([tg.geometry.QuadChunk(c.first_cell, c.num_cells, c.data.float()) for c in field.chunks],
                       field.num_cells, nq, gd, tile)
    xi32, _ = tg.pull_back_block(g32, 0, f32)
    assert np.abs(xi32.to_host_cell_major() - ref[None]).max() < 1e-5


def test_poly_pull_back_freezes_singular_cells(cuda):
    """A cell collapsed to a point: J = 0, K is not finite, the step stays at the largest finite
    value, as the oracle's; its neighbours in the 16-cell group converge."""
    mesh = meshes.cube_box("Hexahedron", 2, 2)
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    g.blocks[0].dofmap[3] = g.blocks[0].dofmap[3, 0]
    pts, _ = tg.refcell.gauss_rule("Hexahedron", 2)
    x = tg.physical_points_block(g, 0, tg.PointSet("Hexahedron", pts, np.ones(len(pts))))
    for precision in ("native", "split"):
        _, step = tg.pull_back_block(g, 0, x, precision=precision)
        s = step.to_host_cell_major()[..., 0]
        assert np.all(s[3] == np.finfo(np.float64).max)
        assert np.delete(s, 3, axis=0).max() <= 1e-13
