"""Grids of a single cell (needs a GPU)."""
import numpy as np
import pytest

import opstream
from equelle_b200.runtime import Runtime
from kernels import launched
from parity import assert_colls
from test_general_form import stiff_exchange

pytestmark = pytest.mark.gpu

GRIDS = [dict(grid_dim=2, nx=1, ny=1, dx=0.7, dy=1.3), dict(grid_dim=3, nx=1, ny=1, nz=1, dx=0.7, dy=1.3, dz=0.5)]


@pytest.mark.parametrize("grid", GRIDS, ids=["2d", "3d"])
def test_operations(gpu_lib, oracle_lib, grid):
    """One cell, no interior face: the oracle's values and Jacobians."""
    got, want = (opstream.op_stream(Runtime(lib, grid)) for lib in (gpu_lib, oracle_lib))
    for k in want:
        assert_colls(got[k], want[k], k)


@pytest.mark.parametrize("grid", GRIDS, ids=["2d", "3d"])
@pytest.mark.parametrize("ncomp", [2, 3])
@pytest.mark.parametrize("coarsest", [1, 128])
def test_systems(gpu_lib, oracle_lib, grid, ncomp, coarsest):
    """Two and three unknowns, whether they count as more than the coarsest
    level or not: within 1e-9 relative of the oracle, in the general form
    (there is no cell of a second colour)."""
    fields = [np.array([0.5 + 0.25 * k]) for k in range(ncomp)]
    params = dict(grid, abs_res_tol=1e-12, linsolver_residual_tolerance=1e-12)
    want = stiff_exchange(Runtime(oracle_lib, params), fields, 0.02, [0.2, 0.4])
    for rep in range(2):
        got, names = launched(gpu_lib, dict(params, linsolver_mg_coarsest=coarsest),
                              lambda er: stiff_exchange(er, fields, 0.02, [0.2, 0.4]))
        assert not any(n.startswith("rb_") for n in names), names
        for g, o in zip(got, want):
            for k in range(ncomp):
                assert np.max(np.abs(g[k] - o[k]) / np.abs(o[k])) <= 1e-9
