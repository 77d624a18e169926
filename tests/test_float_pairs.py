"""Where float pairs stand for the reference's double arithmetic (the
stroker's normals and discriminants, the cubics' quad counts, the mirror tile
mode), the results are the same floats: compared on the CPU over random
values of every scale, zeros and quarter-pixel coordinates."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT, TESTS, _cuda_include


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(TESTS, "_build", "libfloat_pairs.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared",
                        "-I" + _cuda_include(), os.path.join(ROOT, "tests", "float_pairs.cc"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    so = ctypes.CDLL(out)
    so.quad_ends_check.restype = ctypes.c_int64
    return so


@pytest.mark.parametrize("seed", range(3))
def test_pairs_give_the_double_results(lib, seed):
    c = (ctypes.c_int64 * 6)()
    lib.float_pairs_check(ctypes.c_uint32(seed), ctypes.c_int64(1_000_000), c)
    assert list(c[:4]) == [0, 0, 0, 0]
    assert c[5] > 200_000  # the pairs settle them


def test_quad_ends_are_float_divisions(lib):
    assert lib.quad_ends_check(2000) == 0
