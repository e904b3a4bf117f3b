"""The double-float polynomial evaluation (df64 precision of tetrahedra, hexahedra and prisms) against
the f64 polynomial evaluation of the same points, which its own tests hold to the oracle: point sets
without lines, many planes and lines per CTA, ragged counts, outputs at 8-byte addresses, and values its
conversions treat apart (zeros, powers of two, cells scaled far from 1). Bound: 3e-13 of the largest
value, the double-float tests' own."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu

FACTORS = ("points", "jacobian", "detj", "pinv")
CELLS = [("Tetrahedron", 1), ("Tetrahedron", 2), ("Tetrahedron", 3), ("Hexahedron", 1), ("Hexahedron", 2),
         ("Prism", 1), ("Prism", 2)]


def rule_of(cell, kind):
    rng = np.random.default_rng(3)
    if kind == "one":
        return np.full((1, 3), 0.2)
    if kind == "scattered":
        return rng.uniform(0.05, 0.3, size=(7, 3))
    counts = {"rule": (3, 3, 3), "planes": (2, 2, 13), "lines": (2, 40, 1), "large": (9, 9, 9)}[kind]
    pts, _ = tg.refcell.collapsed_rule(cell, counts)
    return pts[rng.permutation(len(pts))] if kind in ("planes", "lines") else pts


def pair(mesh, cell, pts, names=FACTORS, out=None):
    g = tg.Geometry.from_host(mesh, dtype=torch.float64)
    ps = tg.PointSet(cell, pts, np.ones(len(pts)))
    got = tg.geometric_factors_block(g, 0, ps, names, precision="df64", out=out)
    return got, tg.geometric_factors_block(g, 0, ps, names)


def close(got, want, names=FACTORS, tol=3e-13):
    for f in names:
        a, b = got[f].to_host_cell_major(), want[f].to_host_cell_major()
        assert np.abs(a - b).max() <= tol * np.abs(b).max(), f


@pytest.mark.parametrize("kind", ["one", "scattered", "rule", "planes", "lines", "large"])
@pytest.mark.parametrize("cell,degree", CELLS)
def test_point_sets(cuda, cell, degree, kind):
    mesh = meshes.curved_box(cell, 3 if cell == "Hexahedron" else 2, degree, jitter=0.01).first_cells(21)
    pts = rule_of(cell, kind)
    close(*pair(mesh, cell, pts))
    for names in (("points",), ("detj",), ("jacobian", "pinv")):
        close(*pair(mesh, cell, pts, names), names)


@pytest.mark.parametrize("cell,degree", [("Tetrahedron", 2), ("Hexahedron", 2)])
def test_outputs_at_8_byte_addresses(cuda, cell, degree):
    mesh = meshes.curved_box(cell, 3, degree, jitter=0.01).first_cells(21)
    pts = rule_of(cell, "rule")
    out = {}
    for f in FACTORS:
        ln = tg.geometry.FACTOR_LEN[f](3, 3)
        buf = torch.empty(32 * len(pts) * ln + 1, dtype=torch.float64, device="cuda")
        assert buf.data_ptr() % 16 == 0
        out[f] = tg.QuadField([tg.geometry.QuadChunk(0, 21, buf[1:])], 21, len(pts), ln, 16)
    close(*pair(mesh, cell, pts, out=out))


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -40, 2.0 ** 30, 2.0 - 2.0 ** -30])
@pytest.mark.parametrize("cell,degree", [("Hexahedron", 2), ("Tetrahedron", 1), ("Prism", 2)])
def test_zeros_and_powers_of_two(cuda, cell, degree, scale):
    """Axis-aligned cells of side 1/4: J is diagonal or triangular with entries 0 and +-1/4 exactly in both
    (differences of lattice coordinates and products by small integers are exact), at any scale by a power of
    two, and at one whose f32 rounding lands in the next binade."""
    mesh = meshes.cube_box(cell, 4, degree)
    mesh.nodes = mesh.nodes * scale
    got, want = pair(mesh, cell, rule_of(cell, "rule"))
    close(got, want)
    assert np.array_equal(got["jacobian"].to_host_cell_major(), want["jacobian"].to_host_cell_major())


def test_degenerate_cells(cuda):
    """A cell collapsed to a point: det J is 0 and K not finite; the other cells are not disturbed."""
    mesh = meshes.cube_box("Hexahedron", 3, 2)
    cells = mesh.blocks[0].cells.copy()
    cells[4] = cells[4, 0]
    mesh = meshes.HostMesh(3, mesh.nodes, [meshes.HostBlock("Hexahedron", 2, cells)])
    got, want = pair(mesh, "Hexahedron", rule_of("Hexahedron", "rule"))
    d, k = got["detj"].to_host_cell_major(), got["pinv"].to_host_cell_major()
    assert np.all(d[4] == 0.0) and not np.isfinite(k[4]).any()
    keep = np.arange(len(cells)) != 4
    assert np.abs(d[keep] - want["detj"].to_host_cell_major()[keep]).max() <= 3e-13
    assert np.isfinite(k[keep]).all()
