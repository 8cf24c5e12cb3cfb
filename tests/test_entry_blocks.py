"""Jacobian entries around the number that one block of the elementwise and
planned product kernels takes (4 per thread, 1024 per block; needs a GPU)."""
import numpy as np
import pytest

import opstream
from equelle_b200.runtime import Runtime
from parity import assert_colls

pytestmark = pytest.mark.gpu

# cells (entries of a cellwise Jacobian): 1; a part of one entry per thread;
# one block less one, exactly, and one more; several blocks and a remainder.
# The other Jacobians of the stream have 2 to 7 entries a row.
SIZES = [(1, 2, 1), (3, 71, 1), (33, 31, 1), (32, 32, 1), (41, 25, 1), (11, 13, 17)]


@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_entries_across_block_edges(gpu_lib, oracle_lib, nx, ny, nz):
    """Bit for bit the kernels without plans and deferred rules, and the
    oracle's values and Jacobians."""
    grid = dict(grid_dim=3 if nz > 1 else 2, nx=nx, ny=ny, dx=0.7, dy=1.3)
    if nz > 1:
        grid.update(nz=nz, dz=0.5)
    fast = opstream.op_stream(Runtime(gpu_lib, grid))
    generic = opstream.op_stream(Runtime(gpu_lib, dict(grid, stencil_ops=0, spgemm_plan=0, jac_concat=0,
                                                       jac_defer=0)))
    oracle = opstream.op_stream(Runtime(oracle_lib, grid))
    for k in oracle:
        assert_colls(fast[k], generic[k], k, rtol=0.0)
        assert_colls(fast[k], oracle[k], k)
