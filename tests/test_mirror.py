"""The native half of the Python mirror (csrc/mirror.cpp) over the CPU
oracle: operators with collections, numbers and reflected numbers, comparisons
and identity, keyword arguments, the errors of wrong operands, and handles
given back to the library, also from reference cycles."""
import gc
import weakref

import numpy as np
import pytest

from equelle_b200 import capi
from equelle_b200.runtime import Runtime


@pytest.fixture()
def er(oracle_lib):
    return Runtime(oracle_lib, dict(grid_dim=2, nx=8, ny=6))


def test_operators_and_comparisons(er):
    a, b = np.arange(48.0), np.linspace(1.0, 2.0, 48)
    x, y = er.collection(a), er.collection(b)
    for got, want in [(x + y, a + b), (x - y, a - b), (x * y, a * b), (x / y, a / b), (2 + x, 2 + a), (2.5 - x, 2.5 - a),
                      (np.float64(3.0) * x, 3.0 * a), (x * np.float32(3.0), 3.0 * a), (2 / y, 2 / b), (-x, 0.0 - a),
                      (x + "2", a + 2), (er.sqrt(y), np.sqrt(b))]:
        assert np.array_equal(got.value(), want)
    for got, want in [(x < y, a < b), (x <= 5, a <= 5), (5 > x, a < 5), (x >= y, a >= b), (x.eq(5.0), a == 5),
                      (x.ne(y), a != b), (~(x < 5), a >= 5), ((x < 9) & (x > 2), (a < 9) & (a > 2)),
                      ((x < 2) | (x > 9), (a < 2) | (a > 9))]:
        assert np.array_equal(got.values(), want)
    assert (x == x) is True and (x == y) is False and len({x, y, x}) == 2
    assert x.rt is er and isinstance(x.h, int)


def test_methods_take_keywords_and_report_errors(er):
    x = er.collection(np.arange(48.0))
    assert np.array_equal(er.operatorExtend(data=1.5, a=er.allFaces()).value(), np.full(er.info.number_of_faces, 1.5))
    assert len(er.operatorOn(data=x, from_set=er.allCells(), to_set=er.boundaryCells())) == len(er.boundaryCells())
    assert er.maxReduce(x=x) == 47.0 and list(er.spanSubset(x, start=3, num=np.int64(2)).value()) == [3.0, 4.0]
    with pytest.raises(capi.EqgError) as e:
        x + er.collection(np.ones(3))
    assert e.value.code == capi.EQG_ERR_ARG and "size mismatch" in str(e.value)
    for bad in (lambda: x + None, lambda: er.gradient(), lambda: er.trinaryIf(x < 5, x), lambda: er.sqrt(x, y=x)):
        with pytest.raises(TypeError):
            bad()
    with pytest.raises(AttributeError):
        er.gradient(5)
    with pytest.raises(ValueError):
        x + "a"


def test_handles_and_cycles_are_released(oracle_lib):
    class Marker:
        pass

    er = Runtime(oracle_lib, dict(grid_dim=2, nx=4, ny=4))
    er.kept = er.collection(np.ones(16))  # a cycle: the runtime keeps a handle that keeps the runtime
    er.marker = Marker()
    gone = weakref.ref(er.marker)
    del er
    gc.collect()
    assert gone() is None
