"""The two-colour form of the multigrid-preconditioned BiCGStab and the
aggregation along strong directions, at the shapes where they can go wrong:
odd sides (aggregates without some of their black members), sides of 1 and 2,
one direction far stronger than the others (pairs only), 1 x 1 and 2 x 2
blocks, FP64 and FP32-stored preconditioner.  Fields against the FP64 oracle
within the tolerances of the parity tests (the solves' own tolerance, 1e-12
of the right-hand side, is far below them)."""
import numpy as np
import pytest

from equelle_b200 import programs
from equelle_b200.runtime import Runtime

pytestmark = pytest.mark.gpu

SOLVER = dict(abs_res_tol=1e-11, linsolver_residual_tolerance=1e-12, linsolver_max_iterations=5000)


SHAPES = [((19, 7, 5), (10.0, 10.0, 1.0)), ((9, 11, 13), (10.0, 10.0, 10.0)), ((6, 5, 33), (10.0, 10.0, 0.5)),
          ((2, 3, 41), (10.0, 10.0, 2.0)), ((41, 23, None), (10.0, 1.0, 1.0)), ((33, 2, None), (10.0, 10.0, 1.0))]


def two_phase_case(shape, sizes):
    """programs.two_phase_case on cells of another size, with the wells'
    rates for the same part of a cell's pore volume a day."""
    grid, case = programs.two_phase_case(*shape, steps=1)
    case["source_values"] = case["source_values"] * (np.prod(sizes) / (100.0 * (2.0 if shape[2] else 1.0)))
    grid.update(dx=sizes[0], dy=sizes[1])
    if shape[2]:
        grid.update(dz=sizes[2])
    return dict(grid, **SOLVER), case


@pytest.mark.parametrize("shape,sizes", SHAPES)
@pytest.mark.parametrize("precision", ["double", "mixed"])
def test_two_phase_shapes(gpu_lib, oracle_lib, shape, sizes, precision):
    params, case = two_phase_case(shape, sizes)
    for name, fuse in (("fused", 40000), ("launches", 0)):
        eg = Runtime(gpu_lib, dict(params, linsolver_precision=precision, linsolver_mg_fuse_rows=fuse))
        (pg, sg), = programs.two_phase(eg, **case)
        (po, so), = programs.two_phase(Runtime(oracle_lib, params), **case)
        assert np.max(np.abs(sg - so) / np.abs(so)) <= 1e-8, name
        assert np.max(np.abs(pg - po)) <= 1e-8 * np.max(np.abs(po)), name


@pytest.mark.parametrize("nx,ny", [(1, 300), (300, 1), (15, 9), (37, 41), (2, 130)])
def test_heat_shapes(gpu_lib, oracle_lib, nx, ny):
    grid, case = programs.heat_case(nx, ny, steps=2)
    params = dict(grid, abs_res_tol=1e-10, linsolver_residual_tolerance=1e-12)
    got = programs.heat_equation(Runtime(gpu_lib, params), 0.3, 1.0, **case)
    want = programs.heat_equation(Runtime(oracle_lib, params), 0.3, 1.0, **case)
    for g, o in zip(got, want):
        assert np.max(np.abs(g - o) / np.abs(o)) <= 1e-9
