"""Which systems the 32-bit offsets of the device kernels take
(csrc/size_limits.cuh, compiled for the host): cases too large to run in a
test."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "equelle_b200", "csrc")


@pytest.fixture(scope="module")
def limits(tmp_path_factory):
    d = tmp_path_factory.mktemp("limits")
    src, lib = str(d / "limits.cpp"), str(d / "limits.so")
    with open(src, "w") as f:
        f.write('#include "size_limits.cuh"\n'
                'extern "C" int two_colour_fits(int64_t n, int nd, int bb) { return eqg::two_colour_fits(n, nd, bb); }\n'
                'extern "C" int plan_fits(int64_t j, int64_t p) { return eqg::plan_fits(j, p); }\n')
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-o", lib, src])
    h = ctypes.CDLL(lib)
    h.two_colour_fits.argtypes = [ctypes.c_int64, ctypes.c_int, ctypes.c_int]
    h.plan_fits.argtypes = [ctypes.c_int64, ctypes.c_int64]
    return h


@pytest.mark.parametrize("nd,bs", [(6, 2), (4, 2), (6, 1), (4, 1), (6, 3), (4, 3)])
def test_two_colour_form_takes_what_the_general_form_takes(limits, nd, bs):
    """Every cell with its block and those of all neighbours: the stored
    blocks of the general form, whose values need 32-bit offsets."""
    bb = bs * bs
    most = (2**31 - 2) // ((nd + 1) * bb)  # cells whose values number less than 2^31 - 1
    for n in (1, 1000, 2**31 // ((nd + 2) * bb), most):
        assert limits.two_colour_fits(n, nd, bb)
    for n in (most + 1, 2 * most, 2**31 - 1):
        assert not limits.two_colour_fits(n, nd, bb)


def test_plans_number_their_contributions(limits):
    """Products of Jacobians too large for a plan are merged without one: a
    divergence adds every face entry twice, so 2^30 of them (and any more, in
    13 entries a cell as of a gradient of a divergence of a gradient) would
    be 2^31 contributions."""
    for faces in (2**30, 2**30 + 1, 2**31 - 1):
        assert not limits.plan_fits(faces, faces * 13 // 16)
    most = 2**27 - 1
    assert limits.plan_fits(1, 1) and limits.plan_fits(most, 2**30 - 2) and 6 * most < 2**31
    assert not limits.plan_fits(most + 1, 1) and not limits.plan_fits(1, 2**30 - 1)
