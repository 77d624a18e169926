"""The compositor's fast gradient colour against the general one, on the CPU:
every gradient it takes (sorted offsets inside and outside [0, 1], equal and
nearly equal stops, colours past [0, 1]), every tile mode, parameters at the
borders of the stops and of its search cells.  The colours are bytes: equal."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT, TESTS, _cuda_include


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(TESTS, "_build", "libstaged_gradient.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared",
                        "-I" + _cuda_include(), os.path.join(ROOT, "tests", "staged_gradient.cc"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    so = ctypes.CDLL(out)
    so.staged_gradient_check.restype = so.div_by_recip_check.restype = ctypes.c_int64
    so.div_by_recip_check.argtypes = [ctypes.c_uint32, ctypes.c_int64]
    return so


@pytest.mark.parametrize("seed", range(4))
def test_staged_gradient_is_the_general_one(lib, seed):
    n = ctypes.c_int64()
    assert lib.staged_gradient_check(ctypes.c_uint32(seed), 400, ctypes.byref(n)) == 0
    assert n.value > 100000


def test_division_by_reciprocal_is_the_division(lib):
    assert lib.div_by_recip_check(7, 4_000_000) == 0
