"""Python mirror of equelle::EquelleRuntimeCPU over the C ABI.

Same method names and argument meaning as the C++ class generated
simulators use (sintefmath/equelle backends/serial/include/equelle/
EquelleRuntimeCPU.hpp:35-134), so simulators and tests can be written in
the generated style from Python.  Works with any library that exports the
ABI of include/eqg.h: the device runtime (equelle_b200.load_library()) or
the CPU oracle used by the tests.

The handles' operators and the runtime methods of a program's time loop are
native (csrc/mirror.cpp, built into the package as _mirror); what is here
reads results back, makes collections from host arrays and runs the solves.
"""
import ctypes as C

import numpy as np

from . import capi

try:
    from . import _mirror
except ImportError:  # not built yet: a few seconds of the system compiler
    try:
        from . import build
        build.build_mirror()
        from . import _mirror
    except (ImportError, OSError, RuntimeError) as e:
        import warnings
        warnings.warn("the native module equelle_b200._mirror is not built and cannot be built here (%s); runtime "
                      "calls go through ctypes, some ten times the host time each" % (str(e).splitlines() or [""])[0],
                      RuntimeWarning, stacklevel=2)
        from . import _mirror_py as _mirror


class EntitySet(_mirror.SetBase):
    """CollOfCell / CollOfFace."""

    def __len__(self):
        n = C.c_int64()
        self.rt._ok(self.rt.lib.eqg_set_size(self.h, C.byref(n)))
        return n.value

    def size(self):
        return len(self)

    @property
    def entity(self):
        e = C.c_int()
        self.rt._ok(self.rt.lib.eqg_set_entity(self.h, C.byref(e)))
        return e.value

    def indices(self):
        out = np.empty(len(self), dtype=np.int32)
        if out.size:
            self.rt._ok(self.rt.lib.eqg_set_to_host(self.h, out.ctypes.data_as(capi.c_i32_p)))
        return out


class CollOfBool(_mirror.MaskBase):
    """Masks; & | ~ are native."""

    def __len__(self):
        n = C.c_int64()
        self.rt._ok(self.rt.lib.eqg_mask_size(self.h, C.byref(n)))
        return n.value

    def values(self):
        out = np.empty(len(self), dtype=np.uint8)
        if out.size:
            self.rt._ok(self.rt.lib.eqg_mask_to_host(self.h, out.ctypes.data_as(capi.c_u8_p)))
        return out.astype(bool)


class CollOfScalar(_mirror.CollBase):
    """Value plus optional Jacobian (AutoDiffBlock<double>).  Arithmetic
    (equelleTypes.hpp:86-211), negation, < <= > >= and eq(), ne() are native."""

    def __len__(self):
        n = C.c_int64()
        self.rt._ok(self.rt.lib.eqg_coll_size(self.h, C.byref(n)))
        return n.value

    def size(self):
        return len(self)

    def value(self):
        out = np.empty(len(self), dtype=np.float64)
        if out.size:
            self.rt._ok(self.rt.lib.eqg_coll_to_host(self.h, out.ctypes.data_as(capi.c_dbl_p)))
        return out

    def jacobian(self):
        """(rows, cols, rowptr, colind, vals) or None for a constant."""
        r, c, nnz = C.c_int64(), C.c_int64(), C.c_int64()
        self.rt._ok(self.rt.lib.eqg_coll_jacobian_info(self.h, C.byref(r), C.byref(c), C.byref(nnz)))
        if nnz.value < 0:
            return None
        ptr = np.empty(r.value + 1, dtype=np.int64)
        col = np.empty(max(nnz.value, 1), dtype=np.int32)
        val = np.empty(max(nnz.value, 1), dtype=np.float64)
        self.rt._ok(self.rt.lib.eqg_coll_jacobian_to_host(
            self.h, ptr.ctypes.data_as(capi.c_i64_p), col.ctypes.data_as(capi.c_i32_p),
            val.ctypes.data_as(capi.c_dbl_p)))
        return r.value, c.value, ptr, col[:nnz.value], val[:nnz.value]


_mirror.register_classes(CollOfScalar, CollOfBool, EntitySet, capi.EqgError)


class CollOfVector:
    def __init__(self, cols):
        self.cols = list(cols)

    def col(self, i):
        return self.cols[i]

    def numCols(self):
        return len(self.cols)

    def __getitem__(self, i):
        return self.cols[i]

    def __add__(self, o):
        return CollOfVector(a + b for a, b in zip(self.cols, o.cols))

    def __sub__(self, o):
        return CollOfVector(a - b for a, b in zip(self.cols, o.cols))

    def __neg__(self):
        return CollOfVector(-a for a in self.cols)

    def __mul__(self, s):
        return CollOfVector(a * s for a in self.cols)

    __rmul__ = __mul__

    def __truediv__(self, s):
        return CollOfVector(a / s for a in self.cols)


def _addresses(lib):
    """Entry point addresses of a bound library, looked up once per library."""
    table = getattr(lib, "_eqg_addresses", None)
    if table is None:
        table = {n: C.cast(getattr(lib, n), C.c_void_p).value for n in _mirror.entry_points()}
        lib._eqg_addresses = table
    return table


class Runtime(_mirror.RuntimeBase):
    """equelle::EquelleRuntimeCPU over a library exporting include/eqg.h."""

    def __init__(self, lib, params):
        self.lib = lib
        # a class that overrides the methods handles are made through gets them
        # called, by the native methods too
        self._bind(_addresses(lib), any(getattr(type(self), n) is not f for n, f in _PLAIN.items()))
        keys = [str(k).encode() for k in params]
        vals = [str(v).lower() if isinstance(v, bool) else str(v) for v in params.values()]
        vals = [v.encode() for v in vals]
        karr = (C.c_char_p * len(keys))(*keys)
        varr = (C.c_char_p * len(vals))(*vals)
        h = C.c_void_p()
        self._ok(lib.eqg_runtime_create(len(keys), karr, varr, C.byref(h)))
        self.h = h.value
        info = capi.GridInfo()
        self._ok(lib.eqg_runtime_grid_info(self.h, C.byref(info)))
        self.info = info
        self.dimensions = info.dimensions

    def __del__(self):
        h, self.h = getattr(self, "h", None), None
        if h:
            self.lib.eqg_runtime_destroy(h)

    # -- plumbing --------------------------------------------------------
    def _ok(self, status):
        capi.check(self.lib, status)

    def _out(self, fn, cls, *args):
        out = C.c_void_p()
        self._ok(fn(self.h, *args, C.byref(out)))
        return cls(self, out.value)

    def _coll(self, fn, *args):
        return self._out(fn, CollOfScalar, *args)

    def _mask(self, fn, *args):
        return self._out(fn, CollOfBool, *args)

    def _set(self, fn, *args):
        return self._out(fn, EntitySet, *args)

    # -- data in/out -----------------------------------------------------
    def collection(self, values):
        v = np.ascontiguousarray(values, dtype=np.float64)
        return self._coll(self.lib.eqg_coll_from_host, v.ctypes.data_as(capi.c_dbl_p), v.size)

    def constant(self, value, n):
        return self._coll(self.lib.eqg_coll_constant, float(value), int(n))

    def entity_set(self, entity, indices):
        idx = np.ascontiguousarray(indices, dtype=np.int32)
        return self._set(self.lib.eqg_set_from_host, entity, idx.ctypes.data_as(capi.c_i32_p), idx.size)

    def mask(self, values):
        v = np.ascontiguousarray(values, dtype=np.uint8)
        return self._mask(self.lib.eqg_mask_from_host, v.ctypes.data_as(capi.c_u8_p), v.size)

    def variable(self, init):
        return self._coll(self.lib.eqg_variable, init.h)

    # -- topology (index sets, firstCell and secondCell are native) ----------
    def norm(self, x):
        if isinstance(x, EntitySet):
            return self._coll(self.lib.eqg_measure, x.h)
        if isinstance(x, CollOfVector):
            n2 = x.col(0) * x.col(0)
            for d in range(1, x.numCols()):
                n2 = n2 + x.col(d) * x.col(d)
            return self.sqrt(n2)
        return self._coll(self.lib.eqg_unary, capi.ABS, x.h)

    def centroid(self, s):
        return CollOfVector(self._coll(self.lib.eqg_centroid, s.h, d) for d in range(self.dimensions))

    def normal(self, faces):
        return CollOfVector(self._coll(self.lib.eqg_normal, faces.h, d) for d in range(self.dimensions))

    # -- math (gradient, divergence, On, Extend, trinaryIf, sqrt and the
    # reductions are native) ----------------------------------------------
    def dot(self, v1, v2):
        r = v1.col(0) * v2.col(0)
        for d in range(1, self.dimensions):
            r = r + v1.col(d) * v2.col(d)
        return r

    def isEmpty(self, s):
        return self._mask(self.lib.eqg_set_is_empty, s.h)

    # -- solvers ---------------------------------------------------------
    def newtonSolve(self, rescomp, u0):
        err = []

        def tramp(user, u, out):
            try:
                self.lib.eqg_coll_retain(u)
                r = rescomp(CollOfScalar(self, u))
                self.lib.eqg_coll_retain(r.h)
                out[0] = r.h
                return 0
            except Exception as e:  # reported after the C call returns
                err.append(e)
                return 1

        cb = capi.RESIDUAL_FN(tramp)
        out = C.c_void_p()
        st = self.lib.eqg_newton_solve(self.h, cb, None, u0.h, C.byref(out))
        if err:
            raise err[0]
        self._ok(st)
        return CollOfScalar(self, out.value)

    def newtonSolveSystem(self, rescomps, u0s):
        """EquelleRuntimeCPU_impl.hpp:282-339 for any number of blocks."""
        num = [len(u) for u in u0s]
        start = np.concatenate([[0], np.cumsum(num)[:-1]]).astype(int)
        total = int(sum(num))

        start = [int(v) for v in start]

        # Opm::subset(u, ESpan(num, 1, start)) and its inverse, native
        def sub(u, i):
            return self.spanSubset(u, start[i], num[i])

        def sup(x, i):
            return self.spanSuperset(x, start[i], total)

        def combined(u):
            parts = [sub(u, i) for i in range(len(num))]
            res = [f(*parts) for f in rescomps]
            r = sup(res[0], 0)
            for i in range(1, len(res)):
                r = r + sup(res[i], i)
            return r

        u0 = sup(u0s[0], 0)
        for i in range(1, len(u0s)):
            u0 = u0 + sup(u0s[i], i)
        u = self.newtonSolve(combined, u0)
        return tuple(sub(u, i) for i in range(len(num)))

    def solveForUpdate(self, residual):
        return self._coll(self.lib.eqg_solve_for_update, residual.h)

    # -- stats and timing ------------------------------------------------
    def stats(self):
        s = capi.Stats()
        self._ok(self.lib.eqg_runtime_stats(self.h, C.byref(s)))
        return s.as_dict()

    def reset_stats(self):
        self._ok(self.lib.eqg_runtime_reset_stats(self.h))

    def mark(self):
        m = C.c_int()
        self._ok(self.lib.eqg_runtime_mark(self.h, C.byref(m)))
        return m.value

    def elapsed_ms(self, a, b):
        ms = C.c_double()
        self._ok(self.lib.eqg_runtime_elapsed_ms(self.h, a, b, C.byref(ms)))
        return ms.value

    def solve_marks(self, k):
        s, e = C.c_int(), C.c_int()
        self._ok(self.lib.eqg_runtime_solve_marks(self.h, k, C.byref(s), C.byref(e)))
        return s.value, e.value

    def synchronize(self):
        self._ok(self.lib.eqg_runtime_synchronize(self.h))


_PLAIN = {n: vars(Runtime)[n] for n in ("_ok", "_out", "_coll", "_mask", "_set", "constant")}
