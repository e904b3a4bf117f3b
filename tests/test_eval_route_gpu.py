"""f64 evaluation at few points, or of points alone, on meshes that fill the device: the unrolled kernel runs
(bit for bit the loops kernel's values), for every cell that has it; rules of shared lines and small meshes
keep the polynomial kernel. Both agree to rounding."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu

ALL = ("points", "jacobian", "detj", "pinv")
CELLS = [("Tetrahedron", 1, 3), ("Tetrahedron", 2, 3), ("Tetrahedron", 3, 3), ("Hexahedron", 1, 3),
         ("Hexahedron", 2, 3), ("Prism", 1, 3), ("Prism", 2, 3), ("Triangle", 1, 2), ("Triangle", 2, 3),
         ("Triangle", 3, 2), ("Quadrilateral", 1, 3), ("Quadrilateral", 2, 2)]


def mesh_of(cell, degree, gd):
    if gd == 2 or cell in ("Triangle", "Quadrilateral"):
        m = meshes.square_box(cell, 100 if cell == "Triangle" else 140, degree)
        m.nodes = meshes.jitter_interior(m.nodes, m.nodes, 0.0005, 2026)
        return m if gd == 2 else meshes.HostMesh(3, np.concatenate([m.nodes, 0.1 * np.sin(3.0 * m.nodes[:, :1])], 1),
                                                 m.blocks)
    return meshes.curved_box(cell, {"Tetrahedron": 15, "Hexahedron": 27, "Prism": 22}[cell], degree, jitter=0.001)


def run(g, ps, names, strategy="auto"):
    with tg.with_strategy(strategy):
        return {f: v.to_host_cell_major() for f, v in tg.geometric_factors_block(g, 0, ps, names).items()}


@pytest.mark.parametrize("cell,degree,gd", CELLS)
def test_few_points(cuda, cell, degree, gd):
    td = tg.refcell.tdim(cell)
    mesh = mesh_of(cell, degree, gd)
    assert mesh.blocks[0].num_cells >= 128 * 152
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    scattered = np.random.default_rng(3).uniform(0.05, 0.3, size=(3, td))
    for pts, names in ((scattered[:1], ALL), (scattered[:1], ("detj",)), (scattered, ("points",))):
        ps = tg.PointSet(cell, pts, np.ones(len(pts)))
        got, want = run(g, ps, names), run(g, ps, names, "loops")
        for f in names:
            assert np.array_equal(got[f], want[f]), (f, len(pts))
        tile4 = tg.geometric_factors_block(g, 0, ps, names, tile=4, max_chunk_cells=5000)
        assert np.array_equal(tile4[names[0]].to_host_cell_major(), got[names[0]])
    pts, w = tg.refcell.collapsed_rule(cell, (4, 4, 3)[:td])
    ps = tg.PointSet(cell, pts, w)
    got, want = run(g, ps, ALL), run(g, ps, ALL, "loops")
    for f in ALL[:3]:  # (K is the condition number times further off, and jittered P3 triangles reach 1e5)
        assert np.abs(got[f] - want[f]).max() <= 1e-11 * np.abs(want[f]).max(), f
    assert not np.array_equal(got["detj"], want["detj"])  # the polynomial kernel's rounding


def ms(g, ps, names, precision):
    out = tg.geometric_factors_block(g, 0, ps, names, precision=precision)
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            tg.geometric_factors_block(g, 0, ps, names, precision=precision, out=out)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return sorted(times)[3]


@pytest.mark.parametrize("cell,degree,npts", [("Tetrahedron", 2, 24), ("Tetrahedron", 3, 14), ("Hexahedron", 2, 14),
                                              ("Prism", 2, 14)])
def test_double_float_at_scattered_points(cuda, cell, degree, npts):
    """Points that share no line: the double-float path keeps its margin over f64 (0.3 to 0.5 of its time
    measured; the polynomial kernel, whose planes' sums are in FP64, takes longer than f64 there), and its
    error (3e-13 of the largest value)."""
    n = {"Tetrahedron": 28, "Hexahedron": 51, "Prism": 40}[cell]  # 128,000 cells: the device is full
    mesh = meshes.curved_box(cell, n, degree, jitter=0.02 / n)
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    pts = np.random.default_rng(3).uniform(0.05, 0.3, size=(npts, 3))
    ps = tg.PointSet(cell, pts, np.ones(npts))
    for names in (ALL, ("detj",), ("points",)):
        got = tg.geometric_factors_block(g, 0, ps, names, precision="df64")
        want = tg.geometric_factors_block(g, 0, ps, names)
        for f in names:
            a, b = got[f].to_host_cell_major(), want[f].to_host_cell_major()
            assert np.abs(a - b).max() <= 3e-13 * np.abs(b).max(), f
    assert ms(g, ps, ALL, "df64") <= 0.8 * ms(g, ps, ALL, "native")


@pytest.mark.parametrize("precision", ["f32", "split"])
@pytest.mark.parametrize("degree", [1, 2])
def test_hexahedra_in_f32_and_split(cuda, degree, precision):
    """The paired kernel's calls (bit for bit the loops kernel's values): points that share no line, few points,
    points alone, and Q1 with a cell measure, whose sums it forms as it goes. The rest runs the line kernel."""
    g = tg.Geometry.from_host(meshes.curved_box("Hexahedron", 22, degree, jitter=0.001),  # above 64 cells per SM
                              dtype=torch.float32 if precision == "f32" else torch.float64)
    mode = "native" if precision == "f32" else precision
    cells = g.blocks[0].num_cells

    def both(pts, names, measure=False):
        ps = tg.PointSet("Hexahedron", pts, np.full(len(pts), 1.0 / len(pts)))
        res = []
        for strategy in ("auto", "loops"):
            cm = torch.zeros(cells, dtype=torch.float32, device="cuda") if measure else None
            with tg.with_strategy(strategy):
                r = tg.geometric_factors_block(g, 0, ps, names, precision=mode, cell_measure=cm)
            res.append([r[f].to_host_cell_major() for f in names] + ([cm.cpu().numpy()] if measure else []))
        return all(np.array_equal(a, b) for a, b in zip(*res))

    rule = tg.refcell.collapsed_rule("Hexahedron", (3, 3, 3))[0]
    scattered = np.random.default_rng(3).uniform(0.05, 0.95, size=(27, 3))
    assert both(scattered, ALL) and both(rule[:4], ALL) and both(rule, ("points",))
    assert both(rule, ALL, measure=True) == (degree == 1)
    assert not both(rule, ALL)
