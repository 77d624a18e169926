"""The edge sort that ships (edges.cuh), by 32 lanes on the CPU: edges with
equal keys come out in std::sort's order, as the reference sorts them
(sw_raster.cc:679-704), at sizes around the blocks of 16, the lanes and the
on-chip keys, with few and many ties, sorted and reversed input, and inputs
that drive it into the heap sort.  And the bound of the active list that picks
a pass's sweep form, on either side of its counting limit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import TESTS, _cuda_include


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(TESTS, "_build", "libwarp_sort.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared",
                        "-I" + _cuda_include(), os.path.join(TESTS, "warp_sort.cc"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def _same(lib, y, x, dx):
    cols = [np.ascontiguousarray(v, np.int32) for v in (y, x, dx)]
    n = len(cols[0])
    got, want = np.full(n, -1, np.int32), np.full(n, -1, np.int32)
    lib.skc_lanes_sort(*[c.ctypes.data_as(ctypes.c_void_p) for c in cols],
                       got.ctypes.data_as(ctypes.c_void_p), n)
    lib.skc_std_sort_edges(*[c.ctypes.data_as(ctypes.c_void_p) for c in cols],
                           want.ctypes.data_as(ctypes.c_void_p), n)
    assert np.array_equal(got, want), n


@pytest.mark.parametrize("distinct", [1, 2, 3, 40, 1 << 30])
def test_ties_come_out_as_std_sort_leaves_them(lib, distinct):
    rng = np.random.default_rng(distinct)
    for n in list(range(1, 70)) + [95, 96, 97, 128, 200, 383, 384, 385, 1000, 3001]:
        y, x, dx = (rng.integers(-distinct, distinct, n) for _ in range(3))
        _same(lib, y, x, dx)
        _same(lib, np.sort(y), x, dx)
        _same(lib, np.sort(y)[::-1], x * 0, dx)


def test_bad_partitions(lib):
    for n in (100, 384, 385, 2000):
        keys = np.zeros(n, np.int32)
        lib.skc_adversary(keys.ctypes.data_as(ctypes.c_void_p), n)
        zero = np.zeros(n, np.int32)
        _same(lib, keys, zero, zero)
        _same(lib, keys // 3, zero, zero)  # and with ties
        pipe = np.concatenate([np.arange(n // 2), np.arange(n - n // 2)[::-1]])
        _same(lib, pipe, pipe % 2, zero)


def test_active_list_bound(lib):
    rng = np.random.default_rng(9)
    for n in (1, 2, 31, 32, 33, 255, 256, 257, 600, 1500):
        for length in (1, 20, 4000):
            upper = np.sort(rng.integers(0, 1000, n)).astype(np.int32)
            lower = (upper + rng.integers(1, length + 1, n)).astype(np.int32)
            out = np.zeros(2, np.int32)
            lib.skc_max_active(upper.ctypes.data_as(ctypes.c_void_p),
                               lower.ctypes.data_as(ctypes.c_void_p), n,
                               out.ctypes.data_as(ctypes.c_void_p))
            assert out[0] == out[1], (n, length)
