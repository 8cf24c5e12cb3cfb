"""The linear solver's general form, whose V-cycle works on the block graph
over stages: the systems and orderings that the two-colour form does not take
(needs a GPU).  Each test asserts which kernels ran."""
import numpy as np
import pytest

from equelle_b200 import programs
from equelle_b200.runtime import Runtime
from kernels import launched

pytestmark = pytest.mark.gpu

SCALAR = [dict(linsolver_block=0), dict(linsolver_ordering="natural")]


def stiff_exchange(er, fields, eps, timesteps):
    """2 or 3 fields on all cells, implicit in time: diffusion, a small
    fourth-order term (a Laplacian of the Laplacian, which couples cells at
    distance two) and exchange with the next field, solved together."""
    ifaces, all_faces = er.interiorFaces(), er.allFaces()
    trans = er.norm(ifaces) / er.norm(er.centroid(er.firstCell(ifaces)) - er.centroid(er.secondCell(ifaces)))

    def lap(x):
        return er.divergence(er.operatorExtend(trans * er.gradient(x), ifaces, all_faces))

    olds = [er.collection(f) for f in fields]
    n = len(olds)
    out = []
    for dt in timesteps:
        def residual(k, dt=dt, olds=olds):
            def r(*u):
                flow = lap(u[k]) - eps * lap(lap(u[k]))
                return (u[k] - olds[k]) - dt * flow + (0.3 * dt) * (u[k] * u[(k + 1) % n])
            return r

        olds = list(er.newtonSolveSystem([residual(k) for k in range(n)], olds))
        out.append([u.value() for u in olds])
    return out


def _stiff_case(shape, ncomp):
    nx, ny, nz = shape
    grid = dict(grid_dim=2 if nz is None else 3, nx=nx, ny=ny, nz=nz or 1, dx=1.0, dy=1.0, dz=1.0)
    rng = np.random.RandomState(ncomp)
    fields = [0.5 + rng.rand(nx * ny * (nz or 1)) for _ in range(ncomp)]
    return grid, (fields, 0.02, [0.2, 0.4])


def _general(names):
    """The solves took the general form (rb_map is the other form's look at
    the pattern)."""
    assert any(n.startswith("bilu") for n in names), names
    assert not any(n.startswith("rb_") for n in names - {"rb_map"}), names


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("shape,ncomp", [((14, 11, None), 2), ((14, 11, None), 3), ((8, 7, 5), 2), ((6, 5, 4), 3)])
def test_blocks_with_couplings_at_distance_two(gpu_lib, oracle_lib, shape, ncomp, precision):
    """2 x 2 and 3 x 3 blocks: every field within 1e-9 relative of the FP64
    oracle, whether the up-leg goes through A P, recomputes the residual, or
    runs in the fused cycle."""
    grid, args = _stiff_case(shape, ncomp)
    params = dict(grid, abs_res_tol=1e-11, linsolver_residual_tolerance=1e-12, linsolver_max_iterations=5000)
    want = stiff_exchange(Runtime(oracle_lib, params), *args)
    dev = dict(params, linsolver_precision=precision)
    for extra, ran in [(dict(linsolver_mg_fuse_rows=0, linsolver_mg_ap_rows=0), {"mg_correct", "mg_ap_values"}),
                       (dict(linsolver_mg_fuse_rows=0, linsolver_mg_ap_rows=10**9), {"mg_prolong", "mg_residual"}),
                       (dict(linsolver_preconditioner="ilu0"), {"bilu_upper"})]:
        got, names = launched(gpu_lib, dict(dev, **extra), lambda er: stiff_exchange(er, *args))
        _general(names)
        assert ran <= names, (extra, names)
        for step, (g, o) in enumerate(zip(got, want)):
            for k in range(ncomp):
                assert np.max(np.abs(g[k] - o[k]) / np.abs(o[k])) <= 1e-9, (extra, step, k)


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("form", SCALAR, ids=["scalar-blocks", "natural"])
@pytest.mark.parametrize("shape", [(8, 7, 4), (24, 20, None)])
def test_coarse_correction_through_ap_general_form(gpu_lib, oracle_lib, shape, form, precision):
    """Two-phase with 1 x 1 blocks or in natural order: the up-leg through
    A P and the one that recomputes r - A z, within 1e-8 of the oracle."""
    grid, case = programs.two_phase_case(*shape, steps=1)
    params = dict(grid, abs_res_tol=1e-11, linsolver_residual_tolerance=1e-12, linsolver_max_iterations=20000)
    oo = programs.two_phase(Runtime(oracle_lib, params), **case)
    dev = dict(params, linsolver_precision=precision, linsolver_mg_fuse_rows=0, **form)
    for ap_rows, ran in [(0, "mg_correct"), (10**9, "mg_prolong")]:
        og, names = launched(gpu_lib, dict(dev, linsolver_mg_ap_rows=ap_rows), lambda er: programs.two_phase(er, **case))
        _general(names)
        assert ran in names and ("mg_correct" in names) == (ap_rows == 0), names
        for step, ((pg, sg), (po, so)) in enumerate(zip(og, oo)):
            assert np.max(np.abs(sg - so) / np.abs(so)) <= 1e-8, "Sw step %d" % step
            assert np.max(np.abs(pg - po)) <= 1e-8 * np.max(np.abs(po)), "p step %d" % step


def _same_with_fused_levels(gpu_lib, params, program):
    """The cycle's coarse levels in one cluster kernel compute every element
    as the cycle of one launch per step does: the same bits and iteration
    counts with no, some and all levels fused, for cluster sizes 1, 8 and 16,
    and with the smallest levels in block 0's shared memory or not."""
    runs = {}
    for fuse, cluster, local in [(0, 16, 1), (600, 16, 1), (600, 16, 0), (40000, 1, 1), (40000, 8, 1),
                                 (40000, 16, 1), (40000, 16, 0)]:
        p = dict(params, linsolver_mg_fuse_rows=fuse, linsolver_mg_cluster=cluster, linsolver_mg_local=local)
        if (cluster, local) == (16, 1):
            _, names = launched(gpu_lib, p, program)
            _general(names)
            assert ("mg_tail" in names) == (fuse > 0), names
        er = Runtime(gpu_lib, p)
        runs[(fuse, cluster, local)] = (program(er), er.stats()["krylov_iterations"])
    base, its = runs[(0, 16, 1)]
    for key, (out, k) in runs.items():
        assert k == its, key
        for step_a, step_b in zip(out, base):
            for a, b in zip(step_a, step_b):
                assert np.array_equal(a, b), key


@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("shape", [(12, 11, 8), (24, 20, None)])
def test_fused_coarse_cycle_identical_scalar_blocks(gpu_lib, shape, precision):
    grid, case = programs.two_phase_case(*shape, steps=1)
    params = dict(grid, abs_res_tol=1e-10, linsolver_residual_tolerance=1e-10, linsolver_max_iterations=5000,
                  linsolver_precision=precision, linsolver_block=0)
    _same_with_fused_levels(gpu_lib, params, lambda er: programs.two_phase(er, **case))
