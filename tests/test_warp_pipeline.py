"""The dispatch that ships, by 32 lanes on the CPU (tests/warp_pipeline.cc),
against the oracle: each pass by the sweep form its launch takes, two warps a
pass, the lists of 129 to 256 edges among them; passes whose list outgrows
their form; path clips by generation; the row tiles, which cover every pixel
once."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import TESTS, _cuda_include
from skity_gb300 import scene as S
from test_gpu_clip_generations import tree_scene
from test_gpu_sweep_forms import comb_scene

REG64, GENERIC, REG128, REG32, REG256 = range(5)  # kernels.cuh


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(TESTS, "_build", "libwarp_pipeline.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared",
                        "-pthread", "-I" + _cuda_include(),
                        os.path.join(TESTS, "warp_pipeline.cc"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def _render(lib, sc, max_w=1024, slack=0):
    data = sc.to_bytes()
    out = np.zeros((sc.height, sc.width, 4), np.uint8)
    forms = np.zeros(5, np.uint32)
    rc = lib.skc_warp_render(data, ctypes.c_size_t(len(data)), out.ctypes.data_as(ctypes.c_void_p),
                             max_w, slack, forms.ctypes.data_as(ctypes.c_void_p))
    assert rc == 0, rc
    return out, list(forms)


# two active edges a tooth, give or take what a slant adds: the limits of the
# forms, lists of up to 256 and past them, rows wider than the accumulators of
# the 32-edge form and of the others (1,156 and 3,072 pixels)
@pytest.mark.parametrize("teeth,width,height,slant,curved,form", [
    (8, 61, 9, 0.1, False, REG32), (16, 1300, 5, 0.1, True, REG32), (17, 90, 9, 0.1, False, REG64),
    (32, 129, 9, 0.0, True, REG64), (33, 300, 7, 0.0, False, REG128),
    (64, 3200, 5, 0.0, True, REG128), (65, 400, 7, 0.0, False, REG256),
    (100, 500, 7, 0.4, True, REG256), (128, 3200, 5, 0.0, True, REG256),
    (129, 600, 5, 0.0, False, GENERIC)])
@pytest.mark.parametrize("evenodd", [False, True])
def test_forms(lib, oracle_lib, teeth, width, height, slant, curved, form, evenodd):
    sc = comb_scene(teeth, width, height, slant, curved, evenodd)
    got, forms = _render(lib, sc, max_w=100)
    assert forms[form] == 1 and sum(forms) == 1, forms
    assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0


# (a bound above 256 is the generic form's, which takes any list)
@pytest.mark.parametrize("teeth,slack", [(17, 10), (33, 20), (65, 40), (129, 10)])
def test_lists_that_outgrow_their_form(lib, oracle_lib, teeth, slack):
    sc = comb_scene(teeth, 300, 7, 0.0, False, False)
    got, forms = _render(lib, sc, slack=slack)
    assert sum(forms) == 0, forms
    assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0


def test_fills_strokes_and_gradients(lib, oracle_lib):
    sc = S.config2(n_paths=16, width=90, height=70)
    got, forms = _render(lib, sc, max_w=64)
    assert sum(forms) >= 16
    assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0


@pytest.mark.parametrize("groups,depth,off_at", [(1, 4, -1), (3, 2, 1), (2, 3, 2)])
def test_clip_generations(lib, oracle_lib, groups, depth, off_at):
    for op in (S.CLIP_INTERSECT, S.CLIP_DIFFERENCE):
        sc = tree_scene(10 * groups + depth, groups, depth, off_at, op)
        got, _ = _render(lib, sc, max_w=33)
        assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0


@pytest.mark.parametrize("max_w", [32, 100, 1024, 2048])
def test_tiles_cover_every_pixel_once(lib, max_w):
    rng = np.random.default_rng(max_w)
    for n in (1, 2, 30):
        for _ in range(10):
            w = np.exp(rng.uniform(0, np.log(3000), n)).astype(np.uint32)
            h = np.exp(rng.uniform(0, np.log(200), n)).astype(np.uint32)
            p = np.exp(rng.uniform(0, np.log(30000), n)).astype(np.uint32) - 1
            assert lib.skc_tiles_cover(n, *[v.ctypes.data_as(ctypes.c_void_p) for v in (w, h, p)],
                                       max_w) == 0
