"""The coarsest level's inverse at sizes around a warp's rows and columns
(needs a GPU)."""
import numpy as np
import pytest

from equelle_b200 import programs
from equelle_b200.runtime import Runtime

pytestmark = pytest.mark.gpu


# 2 x 2 aggregates: coarsest matrices of 1, 2, 31, 32, 33, 64, 65 and 128 rows
@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 2), (62, 2), (16, 8), (22, 6), (16, 16), (26, 10), (32, 16)])
def test_dense_coarsest_sizes(gpu_lib, oracle_lib, nx, ny):
    """Fields of the FP64 oracle: far within 1e-9 with solves to 1e-12 of the
    right-hand side on matrices whose diagonal dominates."""
    grid, case = programs.heat_case(nx, ny, steps=2)
    params = dict(grid, abs_res_tol=1e-10, linsolver_residual_tolerance=1e-12)
    got = programs.heat_equation(Runtime(gpu_lib, params), 0.3, 1.0, **case)
    want = programs.heat_equation(Runtime(oracle_lib, params), 0.3, 1.0, **case)
    for g, o in zip(got, want):
        assert np.max(np.abs(g - o) / np.abs(o)) <= 1e-9
