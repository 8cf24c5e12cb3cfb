"""The strips of the fused shallow-water stages at their edges: widths around
one and two warps' columns (30), heights around the least strip (8 rows), the
smallest grid, and more rows than one strip takes.  The fused step's fields
are the same bits as those of one kernel per operation."""
import numpy as np
import pytest

from equelle_b200 import programs
from equelle_b200.runtime import Runtime

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (29, 7), (30, 8), (31, 9), (32, 17), (60, 16), (61, 3), (3, 130)])
def test_strip_edges_same_bits(gpu_lib, nx, ny):
    grid, case = programs.swe_case(nx, ny, steps=3, sigma=3.0)
    case["h_init"] = np.where(np.arange(nx * ny) % 7 == 0, 0.01, case["h_init"])  # dry cells among wet ones
    fused = Runtime(gpu_lib, grid)
    got = programs.swe(fused, **case)
    want = programs.swe(Runtime(gpu_lib, dict(grid, fuse=0)), **case)
    assert fused.stats()["fused_evaluations"] > 0
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            assert np.array_equal(a, b)
