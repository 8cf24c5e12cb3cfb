"""The fused shallow-water stages in strips of 16, 32 and 64 rows (smaller
grids all take 8): a ragged grid for each, with a last strip that is nearly
empty in x and cut off in y, and dry cells among the wet ones (needs a GPU).
The fused step's fields are the same bits as those of one kernel per
operation."""
import numpy as np
import pytest

from equelle_b200 import programs
from equelle_b200.runtime import Runtime

pytestmark = pytest.mark.gpu


def _strip_rows(nx, ny):
    """The most rows that give 148 SMs four blocks of four strips of 30
    columns."""
    rows = 64
    while rows > 8 and -(-nx // 30) * -(-ny // rows) < 148 * 4 * 4:
        rows //= 2
    return rows


@pytest.mark.parametrize("nx,ny,rows", [(1501, 1299, 16), (2191, 1901, 32), (3091, 2885, 64)])
def test_tall_strips_same_bits(gpu_lib, nx, ny, rows):
    assert _strip_rows(nx, ny) == rows and nx % 30 == 1 and ny % rows not in (0, 1)
    grid, case = programs.swe_case(nx, ny, steps=2, sigma=40.0)
    case["h_init"] = np.where(np.arange(nx * ny) % 7 == 0, 0.01, case["h_init"])
    fused = Runtime(gpu_lib, grid)
    got = programs.swe(fused, **case)
    want = programs.swe(Runtime(gpu_lib, dict(grid, fuse=0)), **case)
    assert fused.stats()["fused_evaluations"] > 0
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            assert np.array_equal(a, b)
