"""The multigrid hierarchy follows the system that is solved, not the first
one of its pattern: a runtime that has solved other systems gives the fields
and iteration counts of a new one (needs a GPU)."""
import numpy as np
import pytest

from equelle_b200.runtime import Runtime

pytestmark = pytest.mark.gpu

STRONG = 400.0


class Diffusion:
    """Implicit diffusion steps u - u0 - dt div(T grad u) = 0 with one
    transmissibility per direction."""

    def __init__(self, lib, shape, blocks=1, **params):
        nx, ny, nz = shape
        self.n = nx * ny * (nz or 1)
        grid = dict(grid_dim=2 if nz is None else 3, nx=nx, ny=ny, nz=nz or 1, dx=1.0, dy=1.0, dz=1.0)
        self.er = er = Runtime(lib, dict(grid, abs_res_tol=1e-9, linsolver_residual_tolerance=1e-9,
                                         linsolver_max_iterations=5000, **params))
        self.normal = [er.normal(er.interiorFaces()).col(d).value() for d in range(2 if nz is None else 3)]
        self.u0 = [er.collection(np.random.RandomState(k).rand(self.n)) for k in range(blocks)]

    def solve(self, strengths):
        """The fields and the iterations of one solve."""
        er = self.er
        trans = er.collection(sum(s * np.abs(c) for s, c in zip(strengths, self.normal)))

        def residual(k):
            def r(*u):
                flux = er.operatorExtend(trans * er.gradient(u[k]), er.interiorFaces(), er.allFaces())
                return (u[k] - self.u0[k]) - 50.0 * er.divergence(flux) + 0.1 * u[(k + 1) % len(u)]
            return r

        before = er.stats()["krylov_iterations"]
        u = er.newtonSolveSystem([residual(k) for k in range(len(self.u0))], self.u0)
        return [x.value() for x in u], er.stats()["krylov_iterations"] - before


@pytest.mark.parametrize("fuse", [0, 40000])
@pytest.mark.parametrize("blocks", [1, 2])
@pytest.mark.parametrize("shape", [(48, 41, None), (21, 18, 12)])
def test_solves_do_not_depend_on_earlier_ones(gpu_lib, shape, blocks, fuse):
    """Bit for bit the fields and iterations of a runtime of its own, for
    systems strong along one direction after another, without any coupling,
    and back again."""
    dims = 2 if shape[2] is None else 3
    systems = [[STRONG if k == d else 1.0 for k in range(dims)] for d in range(dims)] + [[0.0] * dims, [1.0] * dims]
    fresh = [Diffusion(gpu_lib, shape, blocks, linsolver_mg_fuse_rows=fuse).solve(s) for s in systems]
    used = Diffusion(gpu_lib, shape, blocks, linsolver_mg_fuse_rows=fuse)
    for k in [dims, 0, 1, dims - 1, 0, dims + 1, 1, 1, dims]:
        fields, its = used.solve(systems[k])
        assert its == fresh[k][1], (systems[k], its, fresh[k][1])
        assert all(np.array_equal(a, b) for a, b in zip(fields, fresh[k][0])), systems[k]
