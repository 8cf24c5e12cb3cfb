"""Objects of the Python mirror as a program may meet them besides its plain
runtime calls: before their __init__ has run, with weak references and
attributes, of classes that override the methods handles are made through,
and while other threads run.  Over the CPU oracle."""
import ctypes
import gc
import subprocess
import sys
import threading
import time
import weakref

import numpy as np
import pytest

from conftest import ORACLE_LIB, ROOT
from equelle_b200.runtime import CollOfBool, CollOfScalar, EntitySet, Runtime, _mirror


@pytest.fixture()
def er(oracle_lib):
    return Runtime(oracle_lib, dict(grid_dim=2, nx=8, ny=6))



# every route to a member that __init__ sets, each in a process of its own
# (a crash there is this test's failure, not the end of the run)
BEFORE_INIT = {
    "operand": "x + 1.0", "operand_right": "1.0 - x", "operands": "y + x", "neg": "-x", "compare": "x < 2.0",
    "compare_right": "y < x", "eq": "x.eq(y)", "mask": "~m", "masks": "(y < 2.0) & m", "rt": "x.rt", "h": "x.h",
    "argument": "er.gradient(x)", "extend_over": "er.operatorExtend(1.0, s)", "on": "er.operatorOn(x, s, s)",
    "select": "er.trinaryIf(m, x, x)", "first_cell": "er.firstCell(s)", "reduce": "er.maxReduce(x)",
    "builtin": "early.allCells()", "method": "early.gradient(y)", "sqrt": "early.sqrt(y)",
    "extend": "early.operatorExtend(1.0, er.allCells())", "norm2": "early.twoNorm(y)",
    "span": "early.spanSubset(y, 0, 1)", "runtime_h": "early.h", "bound": "half.allFaces()"}


def test_members_before_init_are_attribute_errors(oracle_lib):
    code = """
import ctypes, sys
import numpy as np
from equelle_b200 import capi
from equelle_b200.runtime import CollOfBool, CollOfScalar, EntitySet, Runtime, _addresses
lib = capi.bind(ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_LOCAL))
er = Runtime(lib, dict(grid_dim=2, nx=8, ny=6))
y = er.collection(np.arange(48.0))
x, m, s = CollOfScalar.__new__(CollOfScalar), CollOfBool.__new__(CollOfBool), EntitySet.__new__(EntitySet)
early, half = Runtime.__new__(Runtime), Runtime.__new__(Runtime)
half.lib = lib
half._bind(_addresses(lib))
try:
    eval(sys.argv[2])
except AttributeError:
    print("attribute error")
"""
    runs = {k: subprocess.Popen([sys.executable, "-c", code, ORACLE_LIB, e], cwd=ROOT, text=True,
                                stdout=subprocess.PIPE, stderr=subprocess.PIPE) for k, e in BEFORE_INIT.items()}
    out = {k: p.communicate() + (p.returncode,) for k, p in runs.items()}
    assert {k: o for k, o in out.items() if o != ("attribute error\n", "", 0)} == {}


def test_handles_take_weak_references_and_attributes(er):
    """As objects of ordinary classes: a weak reference that dies with the
    handle, attributes, and cycles through them."""
    for make in (lambda: er.collection(np.arange(48.0)), lambda: er.mask(np.ones(48)), er.allCells):
        h = make()
        gone = weakref.ref(h)
        h.name = "pressure"
        h.itself = h
        assert h.name == "pressure" and gone() is h
        with pytest.raises(AttributeError):
            h.other
        del h
        gc.collect()
        assert gone() is None
    x = er.collection(np.arange(48.0))
    kept = weakref.WeakValueDictionary(x=x)
    assert np.array_equal((kept["x"] + 1.0).value(), np.arange(48.0) + 1.0)
    del x
    assert "x" not in kept


def test_overridden_plumbing_is_called(oracle_lib):
    """A Runtime subclass that overrides the methods every handle is made
    through sees each call, with the entry point and its arguments; the
    results are those of the plain class."""
    class Traced(Runtime):
        def __init__(self, *args):
            self.calls = []
            super().__init__(*args)

        def _coll(self, fn, *args):
            self.calls.append((fn.__name__, len(args)))
            return super()._coll(fn, *args)

        def _mask(self, fn, *args):
            self.calls.append((fn.__name__, len(args)))
            return super()._mask(fn, *args)

        def _set(self, fn, *args):
            self.calls.append((fn.__name__, len(args)))
            return super()._set(fn, *args)

        def constant(self, value, n):
            self.calls.append(("constant", value, n))
            return super().constant(value, n)

    class Checked(Runtime):
        statuses = []

        def _ok(self, status):
            self.statuses.append(status)
            super()._ok(status)

    grid = dict(grid_dim=2, nx=8, ny=6)

    def stream(er):
        x, cells = er.collection(np.linspace(0.5, 2.0, 48)), er.allCells()
        faces = er.interiorFaces()
        f = er.firstCell(faces)
        m = ~((x < 1.0) & (x < x)) | x.eq(2.0)
        y = er.trinaryIf(m, x + x, 2.0 / x)
        z = er.operatorOn(y, cells, f) * er.sqrt(er.operatorExtend(4.0, faces)) - er.gradient(-y)
        return [m.values(), er.divergence(z).value(), er.spanSuperset(er.spanSubset(y, 3, 4), 1, 9).value(),
                np.array([er.maxReduce(y), er.twoNorm(z)]), er.trinaryIf(m, cells, cells).indices()]

    traced = Traced(oracle_lib, grid)
    got = stream(traced)
    assert traced.calls == [
        ("eqg_coll_from_host", 2), ("eqg_set_builtin", 1), ("eqg_set_builtin", 1), ("eqg_first_cell", 1),
        ("eqg_compare_scalar", 4), ("eqg_compare", 3), ("eqg_mask_logic", 3), ("eqg_mask_logic", 3),
        ("eqg_compare_scalar", 4), ("eqg_mask_logic", 3), ("eqg_binary", 3), ("eqg_binary_scalar", 4),
        ("eqg_select", 3), ("eqg_on", 3), ("constant", 4.0, 7 * 6 + 8 * 5), ("eqg_coll_constant", 2), ("eqg_unary", 2),
        ("eqg_binary", 3), ("eqg_unary", 2), ("eqg_gradient", 1), ("eqg_binary", 3), ("eqg_divergence", 1),
        ("eqg_span_subset", 3), ("eqg_span_superset", 3), ("eqg_set_select", 3)]
    want = stream(Runtime(oracle_lib, grid))
    checked = Checked(oracle_lib, grid)
    for g, c, w in zip(got, stream(checked), want):
        assert np.array_equal(g, w) and np.array_equal(c, w)
    n = len(checked.statuses)
    checked.minReduce(checked.constant(1.0, 3))
    assert checked.statuses[n:] == [0, 0]


@pytest.mark.parametrize("kind", ["coll", "mask", "set"])
def test_handles_are_released_without_the_interpreter_lock(kind):
    """A library's release may take long (the last handle of a destroyed
    runtime waits for its stream): other threads run meanwhile.  The release
    is libc's usleep here, its argument the handle."""
    classes = dict(coll=CollOfScalar, mask=CollOfBool, set=EntitySet)
    usleep = ctypes.cast(ctypes.CDLL(None).usleep, ctypes.c_void_p).value
    er = Runtime.__new__(Runtime)
    er._bind({n: usleep for n in _mirror.entry_points()})
    er.h = None
    started = threading.Event()

    def drop():
        x = classes[kind](er, 900000)
        started.set()
        del x

    t = threading.Thread(target=drop)
    longest, last = 0.0, time.perf_counter()
    t.start()
    started.wait()
    while t.is_alive():
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
        time.sleep(0.001)
    t.join()
    assert longest < 0.45
