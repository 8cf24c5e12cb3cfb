"""The fused shallow-water stages in strips of 1 to 64 rows: a ragged grid for
each, with a last strip that is nearly empty in x and (from 4 rows on) cut off
in y, and dry cells among the wet ones (needs a GPU).  The fused step's fields
are the same bits as those of one kernel per operation."""
import numpy as np
import pytest

from equelle_b200 import programs
from equelle_b200.runtime import Runtime

pytestmark = pytest.mark.gpu


def _strip_rows(nx, ny):
    """The most rows that give 148 SMs four blocks of four strips of 30
    columns; below 8 if all strips are resident (five blocks), 1 if a quarter
    of that is enough."""
    def strips(r):
        return -(-nx // 30) * -(-ny // r)

    rows = 64
    while rows > 8 and strips(rows) < 148 * 4 * 4:
        rows //= 2
    while rows > 1 and strips(rows // 2) <= 148 * 5 * 4 // (1 if rows > 2 else 4):
        rows //= 2
    return rows


@pytest.mark.parametrize("nx,ny,rows", [(61, 47, 1), (31, 370, 1), (31, 373, 2), (271, 283, 2), (511, 507, 4),
                                        (691, 699, 8), (1501, 1299, 16), (2191, 1901, 32), (3091, 2885, 64)])
def test_strips_same_bits(gpu_lib, nx, ny, rows):
    assert _strip_rows(nx, ny) == rows and nx % 30 == 1 and (rows < 4 or ny % rows not in (0, 1))
    grid, case = programs.swe_case(nx, ny, steps=2, sigma=40.0)
    case["h_init"] = np.where(np.arange(nx * ny) % 7 == 0, 0.01, case["h_init"])
    fused = Runtime(gpu_lib, grid)
    got = programs.swe(fused, **case)
    want = programs.swe(Runtime(gpu_lib, dict(grid, fuse=0)), **case)
    assert fused.stats()["fused_evaluations"] > 0
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            assert np.array_equal(a, b)
