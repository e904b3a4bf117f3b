"""Tables whose sections pass 4 GiB: the sections after them stay inside the table's buffer (CPU). Without
a device the call ends at the allocation, with everything before it built and written."""

import os
import pathlib
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
SCRIPT = """
import ctypes
import numpy as np
from gridcl_gb300._lib import lib
n = 1_600_000
pts = np.random.default_rng(0).uniform(size=(n, 3))
h = ctypes.c_void_p()
status = lib().tlg_tables_create(5, 2, 0, 3, 4, pts.ctypes.data_as(ctypes.c_void_p), n, None, ctypes.byref(h))
assert status in (0, 5), (status, lib().tlg_last_error())
if h:
    lib().tlg_tables_destroy(h)
"""


@pytest.mark.skipif(os.sysconf("SC_AVPHYS_PAGES") * os.sysconf("SC_PAGE_SIZE") < 16 << 30, reason="takes 10 GB")
def test_sections_beyond_4_gib():
    """Q2 hexahedra on an f32 mesh at 1.6 million points: the tensor-core sections pass 4 GiB."""
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=dict(os.environ, PYTHONPATH=str(ROOT)),
                       capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-1000:])
