"""Kernels of the linear solver that start while the one before them runs
(needs a GPU)."""
import numpy as np
import pytest

from equelle_b200 import programs
from equelle_b200.runtime import Runtime

pytestmark = pytest.mark.gpu


# fewer rows than a warp; rows that end inside a block, on the level above a
# resident coarse cycle and on levels launched step by step; more blocks than
# the GPU takes at once
@pytest.mark.parametrize("shape,fuse", [((5, 3, None), 0), ((33, 31, None), 0), ((65, 63, None), 600),
                                        ((17, 16, 9), 0), ((17, 16, 9), 600), ((521, 389, None), 40000)])
def test_early_start_matches_one_after_the_other(gpu_lib, shape, fuse):
    """Bit for bit the fields of solves whose kernels run one after the
    other, with as many iterations."""
    grid, case = programs.two_phase_case(*shape, steps=1)
    runs = []
    for pdl in (0, 1):
        eg = Runtime(gpu_lib, dict(grid, abs_res_tol=1e-10, linsolver_residual_tolerance=1e-10,
                                   linsolver_max_iterations=5000, linsolver_mg_fuse_rows=fuse, linsolver_pdl=pdl))
        (p, s), = programs.two_phase(eg, **case)
        runs.append((p, s, eg.stats()["krylov_iterations"]))
    assert runs[0][2] == runs[1][2]
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
