"""Values computed in the launch of their Jacobian, and apart where there are
many rows (needs a GPU)."""
import numpy as np
import pytest

import opstream
from equelle_b200.runtime import Runtime
from parity import assert_colls

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 1), (37, 28), (32, 32)])
def test_values_of_small_collections(gpu_lib, oracle_lib, nx, ny):
    """Values that run beside Jacobians are those of the same operations on
    collections without Jacobians, bit for bit, on one cell and around the
    1024 rows of a block; both are the oracle's."""
    grid = dict(grid_dim=2, nx=nx, ny=ny, dx=0.7, dy=1.3)
    out = {}
    for name, lib in (("gpu", gpu_lib), ("oracle", oracle_lib)):
        er = Runtime(lib, grid)
        n = nx * ny
        rng = np.random.default_rng(5)
        a, b = rng.uniform(-2.0, 2.0, n), rng.uniform(0.5, 2.0, n)
        a[0] = np.inf if n > 2 else a[0]
        for ad in (True, False):
            u, v = er.collection(a), er.collection(b)
            if ad:
                u, v = er.variable(u), er.variable(v)
            m = u > v
            res = [u + v, u - v, u * v, u / v, er.trinaryIf(m, u, v)]
            out[name, ad] = [x.value() for x in res]
    for k in range(5):
        assert np.array_equal(out["gpu", True][k], out["gpu", False][k], equal_nan=True)
        assert np.array_equal(out["gpu", True][k], out["oracle", True][k], equal_nan=True)


def test_values_of_many_rows(gpu_lib, oracle_lib):
    """More rows than are taken along (2^19), against the oracle."""
    grid = dict(grid_dim=2, nx=1024, ny=520, dx=0.7, dy=1.3)
    got, want = (opstream.op_stream(Runtime(lib, grid)) for lib in (gpu_lib, oracle_lib))
    for k in ("add_ad", "sub_ad", "mul", "div_ad"):
        assert_colls(got[k], want[k], k)
