"""Coarsest levels of 1, 2, 31, 32, 33, 64 and 65 rows (warps of the dense
inverse without, with some and with all of their rows and columns), and
levels of fewer rows than a warp, in the two-colour form (needs a GPU).
Coarsening to such sizes takes a small linsolver_mg_coarsest."""
import numpy as np
import pytest

from equelle_b200 import programs
from equelle_b200.runtime import Runtime
from kernels import launched
from test_gpu_parity import reaction_diffusion3

pytestmark = pytest.mark.gpu


def _two_colour_multigrid(names, fuse):
    """The solves took the two-colour form's V-cycle, without the fallback."""
    assert {"rb_factor_black", "rb_spmv_omega"} <= names and not any(n.startswith(("bilu", "mg_tail")) for n in names)
    assert ("rb_tail" in names) == (fuse > 0) and ("rb_dense" in names) == (fuse == 0)


def _coarsest(nx, ny, most):
    while nx * ny > most:
        nx, ny = (nx + 1) // 2, (ny + 1) // 2
    return nx * ny


@pytest.mark.parametrize("fuse", [0, 40000])
@pytest.mark.parametrize("nx,ny,rows", [(61, 2, 1), (61, 2, 2), (61, 2, 31), (64, 2, 32), (65, 2, 33), (32, 32, 64),
                                        (10, 26, 65)])
def test_inverses_of_small_coarsest_levels(gpu_lib, oracle_lib, nx, ny, rows, fuse):
    """Fields of the FP64 oracle: far within 1e-9 with solves to 1e-12 of the
    right-hand side on matrices whose diagonal dominates."""
    assert _coarsest((nx + 1) // 2, (ny + 1) // 2, rows) == rows
    grid, case = programs.heat_case(nx, ny, steps=2)
    params = dict(grid, abs_res_tol=1e-10, linsolver_residual_tolerance=1e-12)
    got, names = launched(gpu_lib, dict(params, linsolver_mg_coarsest=rows, linsolver_mg_fuse_rows=fuse),
                          lambda er: programs.heat_equation(er, 0.3, 1.0, **case))
    _two_colour_multigrid(names, fuse)
    want = programs.heat_equation(Runtime(oracle_lib, params), 0.3, 1.0, **case)
    for g, o in zip(got, want):
        assert np.max(np.abs(g - o) / np.abs(o)) <= 1e-9


@pytest.mark.parametrize("fuse", [0, 40000])
@pytest.mark.parametrize("shape", [(5, 3, None), (3, 2, 2), (2, 1, None), (1, 7, None), (9, 5, 3)])
def test_levels_of_fewer_rows_than_a_warp(gpu_lib, oracle_lib, shape, fuse):
    """Two-phase (2 x 2 blocks) down to a single cell: within 1e-8 of the
    oracle, and bit for bit the fields of kernels that run one after the
    other (linsolver_pdl=0)."""
    grid, case = programs.two_phase_case(*shape, steps=1)
    params = dict(grid, abs_res_tol=1e-11, linsolver_residual_tolerance=1e-12, linsolver_max_iterations=5000)
    small = dict(params, linsolver_mg_coarsest=2, linsolver_mg_fuse_rows=fuse)
    _, names = launched(gpu_lib, small, lambda er: programs.two_phase(er, **case))
    _two_colour_multigrid(names, fuse)
    (po, so), = programs.two_phase(Runtime(oracle_lib, params), **case)
    runs = []
    for pdl in (0, 1):
        (p, s), = programs.two_phase(Runtime(gpu_lib, dict(small, linsolver_pdl=pdl)), **case)
        assert np.max(np.abs(s - so) / np.abs(so)) <= 1e-8
        assert np.max(np.abs(p - po)) <= 1e-8 * np.max(np.abs(po))
        runs.append((p, s))
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])


@pytest.mark.parametrize("fuse", [0, 40000])
def test_three_species_down_to_one_cell(gpu_lib, oracle_lib, fuse):
    """3 x 3 blocks: every species within 1e-9 relative of the oracle."""
    grid = dict(grid_dim=3, nx=7, ny=5, nz=3, dx=1.0, dy=1.0, dz=1.0)
    rng = np.random.RandomState(3)
    fields = [1.0 + rng.rand(105), 0.5 + rng.rand(105), 0.1 * rng.rand(105)]
    args = (fields, (2.0, 0.5, (1.0, 0.3, 0.05)), [0.1, 0.2])
    params = dict(grid, abs_res_tol=1e-12, linsolver_residual_tolerance=1e-12, linsolver_max_iterations=5000)
    got, names = launched(gpu_lib, dict(params, linsolver_mg_coarsest=3, linsolver_mg_fuse_rows=fuse),
                          lambda er: reaction_diffusion3(er, *args))
    _two_colour_multigrid(names, fuse)
    want = reaction_diffusion3(Runtime(oracle_lib, params), *args)
    for g, o in zip(got, want):
        for k in range(3):
            assert np.max(np.abs(g[k] - o[k]) / np.abs(o[k])) <= 1e-9
