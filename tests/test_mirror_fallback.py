"""The Python mirror where its native module is neither built nor buildable:
the same classes over ctypes.  In a process that cannot import the module and
whose compiler is missing, over the CPU oracle."""
import subprocess
import sys

from conftest import ORACLE_LIB, ROOT

BLOCKED = """
import ctypes, sys, warnings
class NoNativeModule:
    def find_spec(self, name, path=None, target=None):
        if name == "equelle_b200._mirror":
            raise ImportError("no module named " + name)
sys.meta_path.insert(0, NoNativeModule())
from equelle_b200 import build, capi
build.CXX = "/nonexistent/g++"
build._stale = lambda target, sources: True
with warnings.catch_warnings(record=True) as caught:
    warnings.simplefilter("always")
    from equelle_b200 import runtime
assert [w.category for w in caught] == [RuntimeWarning]
assert runtime._mirror.__name__ == "equelle_b200._mirror_py"
"""


def _run(code, *args):
    p = subprocess.run([sys.executable, "-c", BLOCKED + code, *args], cwd=ROOT, text=True, capture_output=True)
    assert p.returncode == 0, p.stdout + p.stderr


def test_same_results_and_errors_without_the_native_module(oracle_lib):
    """The operators, methods and errors that the native module is tested
    with, and a program with Newton solves."""
    _run("""
sys.path.insert(0, "tests")
import pytest
sys.exit(pytest.main(["-q", "-p", "no:cacheprovider", "tests/test_mirror.py", "tests/test_oracle_golden.py",
                      "-m", "not gpu"]))
""")


def test_program_without_the_native_module(oracle_lib):
    _run("""
import numpy as np
from equelle_b200 import programs
lib = capi.bind(ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_LOCAL))
grid, case = programs.two_phase_case(5, 4, steps=1)
(p, s), = programs.two_phase(runtime.Runtime(lib, grid), **case)
grid, case = programs.swe_case(7, 5, steps=2)
w, hu, hv = programs.swe(runtime.Runtime(lib, grid), **case)[-1]
assert all(np.isfinite(x).all() for x in (p, s, w, hu, hv)) and s.max() > 0.2
""", ORACLE_LIB)
