"""What csrc/mirror.cpp (the module _mirror) provides, in Python over ctypes:
for interpreters that the native module is not built for and cannot be built
for (no compiler or Python headers, a package that cannot be written to).
Same classes, methods and errors; a runtime call takes 2 to 4 us of
interpreter work where the native one takes 0.2.
"""
import ctypes as C

from . import capi


def register_classes(coll, mask, entity_set, error):
    pass


def entry_points():
    return ()


class _Handle:
    _release = None

    def __init__(self, rt, h):
        self.rt = rt
        self.h = h

    def __del__(self):
        h = getattr(self, "h", None)
        if h:
            self.h = None
            getattr(self.rt.lib, self._release)(h)


class SetBase(_Handle):
    _release = "eqg_set_release"


class MaskBase(_Handle):
    _release = "eqg_mask_release"

    def _logic(self, op, other):
        return self.rt._mask(self.rt.lib.eqg_mask_logic, op, self.h, other.h if other is not None else None)

    def __and__(self, o):
        return self._logic(capi.AND, o)

    def __or__(self, o):
        return self._logic(capi.OR, o)

    def __invert__(self):
        return self._logic(capi.NOT, None)


class CollBase(_Handle):
    _release = "eqg_coll_release"

    def _bin(self, op, other, reflected=False):
        rt = self.rt
        if isinstance(other, CollBase):
            a, b = (other, self) if reflected else (self, other)
            return rt._coll(rt.lib.eqg_binary, op, a.h, b.h)
        return rt._coll(rt.lib.eqg_binary_scalar, op, self.h, float(other), 1 if reflected else 0)

    def __add__(self, o):
        return self._bin(capi.ADD, o)

    def __radd__(self, o):
        return self._bin(capi.ADD, o, True)

    def __sub__(self, o):
        return self._bin(capi.SUB, o)

    def __rsub__(self, o):
        return self._bin(capi.SUB, o, True)

    def __mul__(self, o):
        return self._bin(capi.MUL, o)

    def __rmul__(self, o):
        return self._bin(capi.MUL, o, True)

    def __truediv__(self, o):
        return self._bin(capi.DIV, o)

    def __rtruediv__(self, o):
        return self._bin(capi.DIV, o, True)

    def __neg__(self):
        return self.rt._coll(self.rt.lib.eqg_unary, capi.NEG, self.h)

    def _cmp(self, op, other):
        rt = self.rt
        if isinstance(other, CollBase):
            return rt._mask(rt.lib.eqg_compare, op, self.h, other.h)
        return rt._mask(rt.lib.eqg_compare_scalar, op, self.h, float(other), 0)

    def __lt__(self, o):
        return self._cmp(capi.LT, o)

    def __le__(self, o):
        return self._cmp(capi.LE, o)

    def __gt__(self, o):
        return self._cmp(capi.GT, o)

    def __ge__(self, o):
        return self._cmp(capi.GE, o)

    def eq(self, o):
        return self._cmp(capi.EQ, o)

    def ne(self, o):
        return self._cmp(capi.NE, o)


class RuntimeBase:
    def _bind(self, addresses, hooked=False):
        pass

    def allCells(self):
        return self._set(self.lib.eqg_set_builtin, capi.ALL_CELLS)

    def boundaryCells(self):
        return self._set(self.lib.eqg_set_builtin, capi.BOUNDARY_CELLS)

    def interiorCells(self):
        return self._set(self.lib.eqg_set_builtin, capi.INTERIOR_CELLS)

    def allFaces(self):
        return self._set(self.lib.eqg_set_builtin, capi.ALL_FACES)

    def boundaryFaces(self):
        return self._set(self.lib.eqg_set_builtin, capi.BOUNDARY_FACES)

    def interiorFaces(self):
        return self._set(self.lib.eqg_set_builtin, capi.INTERIOR_FACES)

    def firstCell(self, faces):
        return self._set(self.lib.eqg_first_cell, faces.h)

    def secondCell(self, faces):
        return self._set(self.lib.eqg_second_cell, faces.h)

    def sqrt(self, x):
        return self._coll(self.lib.eqg_unary, capi.SQRT, x.h)

    def gradient(self, x):
        return self._coll(self.lib.eqg_gradient, x.h)

    def negGradient(self, x):
        return self._coll(self.lib.eqg_neg_gradient, x.h)

    def divergence(self, x):
        return self._coll(self.lib.eqg_divergence, x.h)

    def interiorDivergence(self, x):
        return self._coll(self.lib.eqg_interior_divergence, x.h)

    def operatorExtend(self, data, a, b=None):
        if b is None:
            return self.constant(data, len(a))
        if isinstance(data, SetBase):
            return self._set(self.lib.eqg_set_extend, data.h, a.h, b.h)
        return self._coll(self.lib.eqg_extend, data.h, a.h, b.h)

    def operatorOn(self, data, from_set, to_set):
        if isinstance(data, SetBase):
            return self._set(self.lib.eqg_set_on, data.h, from_set.h, to_set.h)
        return self._coll(self.lib.eqg_on, data.h, from_set.h, to_set.h)

    def trinaryIf(self, pred, a, b):
        if isinstance(a, SetBase):
            return self._set(self.lib.eqg_set_select, pred.h, a.h, b.h)
        return self._coll(self.lib.eqg_select, pred.h, a.h, b.h)

    def _reduce(self, op, x):
        r = C.c_double()
        self._ok(self.lib.eqg_reduce(self.h, op, x.h, C.byref(r)))
        return r.value

    def minReduce(self, x):
        return self._reduce(capi.MIN, x)

    def maxReduce(self, x):
        return self._reduce(capi.MAX, x)

    def sumReduce(self, x):
        return self._reduce(capi.SUM, x)

    def prodReduce(self, x):
        return self._reduce(capi.PROD, x)

    def twoNorm(self, x):
        r = C.c_double()
        self._ok(self.lib.eqg_two_norm(self.h, x.h, C.byref(r)))
        return r.value

    def spanSubset(self, u, start, num):
        return self._coll(self.lib.eqg_span_subset, u.h, int(start), int(num))

    def spanSuperset(self, u, start, total):
        return self._coll(self.lib.eqg_span_superset, u.h, int(start), int(total))
