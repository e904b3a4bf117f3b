"""A point set with a coordinate that is not finite: its point gets what the tabulation gives it (NaN), and
the other points keep their values, whichever kernel the rest of the rule would run."""

import numpy as np
import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu

FACTORS = ("points", "jacobian", "detj", "pinv")
TOL = {"native": 1e-12, "df64": 3e-13, "split": 1e-5, "f32": 1e-4}  # of the largest value, curved cells


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("at", [0, 5])
@pytest.mark.parametrize("cell,degree,precision",
                         [("Tetrahedron", 2, "native"), ("Hexahedron", 2, "native"), ("Prism", 1, "native"),
                          ("Triangle", 2, "native"), ("Quadrilateral", 1, "native"), ("Tetrahedron", 3, "df64"),
                          ("Hexahedron", 2, "df64"), ("Hexahedron", 2, "split"), ("Hexahedron", 1, "f32")])
def test_one_bad_coordinate(cuda, cell, degree, precision, at, value):
    td = tg.refcell.tdim(cell)
    if td == 2:
        mesh = meshes.square_box(cell, 4, degree).first_cells(21)
    else:
        mesh = meshes.curved_box(cell, 3 if cell == "Hexahedron" else 2, degree, jitter=0.01).first_cells(21)
    pts, _ = tg.refcell.collapsed_rule(cell, (3, 3, 3)[:td])
    g = tg.Geometry.from_host(mesh, dtype=torch.float32 if precision == "f32" else torch.float64)
    mode = "native" if precision == "f32" else precision
    want = tg.geometric_factors_block(g, 0, tg.PointSet(cell, pts, np.ones(len(pts))), FACTORS, precision=mode)
    bad = pts.copy()
    bad[at, td - 1] = value
    got = tg.geometric_factors_block(g, 0, tg.PointSet(cell, bad, np.ones(len(pts))), FACTORS, precision=mode)
    keep = np.arange(len(pts)) != at
    for f in FACTORS:
        a, b = got[f].to_host_cell_major(), want[f].to_host_cell_major()
        assert np.abs(a[:, keep] - b[:, keep]).max() <= TOL[precision] * np.abs(b).max(), f
        if f == "points":
            assert not np.isfinite(a[:, at]).all(axis=-1).any()
