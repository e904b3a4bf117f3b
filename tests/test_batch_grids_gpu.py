"""The batch tuner offers grids to the blocks whose kernel takes one, and only to them: the polynomial kernels
launch a CTA per group of cells whatever the choice (a grid returned for such a block would be noise between
identical launches)."""

import pytest
import torch

import gridcl_gb300 as tg
from gridcl_gb300 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,degree,precision", [("Tetrahedron", 2, "native"), ("Hexahedron", 2, "native"),
                                                   ("Prism", 1, "native"), ("Hexahedron", 1, "df64")])
def test_no_grid_where_none_applies(cuda, cell, degree, precision):
    for n in (2, 3, 5):
        g = tg.Geometry.from_host(meshes.curved_box(cell, n, degree, jitter=0.01), dtype=torch.float64)
        for order in (3, 4, 5):
            batch = tg.Batch(g, tg.QuadRule.for_grid(g, order), precision=precision)
            assert batch.tune() == [0], (n, order)
