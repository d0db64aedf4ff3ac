"""Host conversions of the integer pair sweeps (csrc/px_units.h), compiled for
this machine: the squared cut-off in units of r2.  Whole numbers: no tolerance."""
import ctypes as C
import math
import os
import subprocess

import pytest

from mdynamix_gb300.build import CSRC


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("px")
    src, so = d / "px.cpp", d / "px.so"
    src.write_text('#include "px_units.h"\n'
                   'extern "C" unsigned long long cut2(double rc2, int rho) '
                   '{ return px_cut2(rc2, rho); }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    L = C.CDLL(os.fspath(so))
    L.cut2.argtypes, L.cut2.restype = [C.c_double, C.c_int], C.c_uint64
    return L


@pytest.mark.parametrize("rho", [2, 3, 4, 5])
def test_no_cutoff_keeps_every_pair(lib, rho):
    """Without a skin the cut-off is 1e300 (mdx_set_params): above every r2, which
    is below 3 2^60."""
    for rc2 in (1e300, 1e100, float("inf")):
        assert lib.cut2(rc2, rho) >= 3 << 60, rc2


@pytest.mark.parametrize("rho", [2, 3, 4, 5])
def test_cutoff_in_units_of_r2(lib, rho):
    for rc in (2.5, 9.0, 12.0, 30.999):
        want = math.floor(math.ldexp(rc * rc, 60 - 2 * rho))
        if want < 3 << 60:
            assert lib.cut2(rc * rc, rho) == want
        else:  # every |d| < 2^rho is inside
            assert lib.cut2(rc * rc, rho) >= 3 << 60
