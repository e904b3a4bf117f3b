"""Point sets whose tables take the polynomial kernels' dynamic shared memory to just below 48 KiB, where
the static bytes beside it pass the default limit: each is evaluated in a process of its own (an earlier
larger launch would have raised a kernel's limit) and held to the loops kernel."""

import os
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]
SCRIPT = """
import sys
import numpy as np, torch
import gridcl_gb300 as tg
from gridcl_gb300 import meshes
cell, degree, precision = sys.argv[1], int(sys.argv[2]), sys.argv[3]
pts, w = tg.refcell.collapsed_rule(cell, tuple(int(c) for c in sys.argv[4].split("x")))
g = tg.Geometry.from_host(meshes.curved_box(cell, 2, degree, jitter=0.01), dtype=torch.float64)
ps = tg.PointSet(cell, pts, w)
names = ("points", "jacobian", "detj", "pinv")
got = tg.geometric_factors_block(g, 0, ps, names, precision=precision)
with tg.with_strategy("loops"):
    want = tg.geometric_factors_block(g, 0, ps, names)
for f in names:
    a, b = got[f].to_host_cell_major(), want[f].to_host_cell_major()
    assert np.abs(a - b).max() <= 3e-13 * np.abs(b).max(), f
"""


# (dynamic bytes: 48960 beside 400 static ones, 48864 beside 400, 49152 beside the barrier's, twice)
@pytest.mark.parametrize("cell,degree,precision,rule",
                         [("Tetrahedron", 2, "df64", "7x7x7"), ("Prism", 2, "df64", "8x3x3"),
                          ("Tetrahedron", 1, "native", "5x8x12"), ("Tetrahedron", 2, "native", "12x11x4")])
def test_sizes_just_below_the_default_limit(cuda, cell, degree, precision, rule):
    r = subprocess.run([sys.executable, "-c", SCRIPT, cell, str(degree), precision, rule], cwd=ROOT,
                       env=dict(os.environ, PYTHONPATH=str(ROOT)), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
