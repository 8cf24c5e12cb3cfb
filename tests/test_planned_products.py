"""Operator products around the 2^17 entries up to which a thread takes one
entry of the product (needs a GPU)."""
import numpy as np
import pytest

from equelle_b200.runtime import Runtime
from parity import assert_colls

pytestmark = pytest.mark.gpu


# a gradient has two entries per interior face: 2 less than the line, the line
# and 2 more; the last case's divergence (129,340 entries) is below it
@pytest.mark.parametrize("nx,ny,entries", [(1, 65536, 2**17 - 2), (2, 21846, 2**17), (123, 268, 2**17 + 2),
                                           (130, 200, 2 * (2 * 26000 - 330))])
def test_products_around_the_line(gpu_lib, oracle_lib, nx, ny, entries):
    """Gradients, divergences and extensions, also of Jacobians with
    deferred rules: the oracle's values and Jacobians, and bit for bit those of
    the merge without plans."""
    grid = dict(grid_dim=2, nx=nx, ny=ny, dx=0.7, dy=1.3)
    out = []
    for lib, extra in ((gpu_lib, {}), (gpu_lib, dict(spgemm_plan=0)), (oracle_lib, {})):
        er = Runtime(lib, dict(grid, **extra))
        rng = np.random.default_rng(1)
        u = er.variable(er.collection(rng.uniform(0.5, 1.5, nx * ny)))
        t = er.collection(rng.uniform(0.1, 1.0, er.info.number_of_interior_faces))
        g = er.gradient(u)
        f = er.operatorExtend(t * er.gradient(u * u), er.interiorFaces(), er.allFaces())
        out.append(dict(grad=g, ext=f, div=er.divergence(f), div_deferred=er.divergence(t * g)))
    assert out[0]["grad"].jacobian()[4].size == entries
    for k in out[0]:
        assert_colls(out[0][k], out[1][k], k, rtol=0.0)
        assert_colls(out[0][k], out[2][k], k)
