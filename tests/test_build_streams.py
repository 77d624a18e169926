"""The threaded stream build (BuildStreams: runs of canvases parsed on host
threads, then appended with their indices and offsets moved) builds the
same batch, byte for byte, as one thread adding the canvases in order --
over scenes with every kind of record a stream holds: gradients of each
kind, strokes, colour filters, blur temp canvases, layers, path clips and
images."""
import ctypes

import pytest

from skity_gb300 import scene as S


def _streams():
    from test_image_shader import image_scene
    from test_oracle_pin import (blend_modes_scene, blur_styles_scene, clip_path_cases_scene,
                                 clipped_scene, color_filters_scene, path_clips_scene,
                                 sweep_conical_scene, translated_scene)
    scenes = list(S.config3(n_canvases=24, scale=0.2))
    scenes += [translated_scene(), clipped_scene(), blend_modes_scene(), sweep_conical_scene(),
               blur_styles_scene(), color_filters_scene(), path_clips_scene(),
               clip_path_cases_scene(), image_scene(),
               S.layered_scene(S.SEED_BASE + 420, 96, 80, 60, 3),
               S.config4(n_outlines=400, width=256, height=256, blur_frac=0.3),
               S.config2(n_paths=300, width=256, height=256)]
    # the feature scenes spread between the plain canvases, so runs mix both
    mixed = []
    for i, sc in enumerate(scenes[24:]):
        mixed += scenes[2 * i:2 * i + 2] + [sc]
    return [sc.to_bytes() for sc in mixed]


@pytest.mark.parametrize("threads", [2, 3, 8, 16])
def test_threaded_build_matches_one_thread(cpu_pipeline, threads):
    lib = cpu_pipeline
    lib.skc_build_streams_compare.argtypes = [ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p,
                                              ctypes.c_uint]
    bufs = _streams()
    n = len(bufs)
    cbufs = [ctypes.create_string_buffer(b, len(b)) for b in bufs]
    ptrs = (ctypes.c_void_p * n)(*[ctypes.addressof(c) for c in cbufs])
    lens = (ctypes.c_size_t * n)(*[len(b) for b in bufs])
    assert lib.skc_build_streams_compare(n, ptrs, lens, threads) == 0


def test_threaded_build_reports_first_bad_stream(cpu_pipeline):
    """A malformed stream fails the build with the status the one-thread
    loop returns for the first bad stream in order."""
    lib = cpu_pipeline
    lib.skc_build_streams_compare.argtypes = [ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p,
                                              ctypes.c_uint]
    bufs = [sc.to_bytes() for sc in S.config3(n_canvases=16, scale=0.1)]
    bufs[9] = bufs[9][:len(bufs[9]) // 2]  # truncated
    n = len(bufs)
    cbufs = [ctypes.create_string_buffer(b, len(b)) for b in bufs]
    ptrs = (ctypes.c_void_p * n)(*[ctypes.addressof(c) for c in cbufs])
    lens = (ctypes.c_size_t * n)(*[len(b) for b in bufs])
    assert lib.skc_build_streams_compare(n, ptrs, lens, 4) == -2  # INVALID_ARGUMENT


def _one_large(draws, bad=None):
    """One canvas of `draws` draws of 48 verbs: solids, gradients of each kind,
    image shaders, strokes, colour filters, blurs of each style, path clips."""
    import numpy as np
    rng = np.random.default_rng(draws)
    b = S.SceneBuilder(300, 200)
    img = b.add_image(rng.integers(0, 256, (5, 7, 4), dtype=np.uint8), S.ALPHA_UNPREMUL)
    square = [S.MOVE, S.LINE, S.LINE, S.LINE, S.CLOSE]
    for i in range(draws):
        verbs = [S.MOVE] + [[S.LINE, S.QUAD, S.CUBIC][j % 3] for j in range(46)] + [S.CLOSE]
        npts = 1 + sum({S.LINE: 1, S.QUAD: 2, S.CUBIC: 3}[v] for v in verbs[1:-1])
        pts = rng.uniform(-10, [310, 210], (npts, 2)).astype(np.float32)
        p = S.default_paint()
        p["style"] = i % 4
        p["stroke_width"] = 2.5
        p["fill_color"] = tuple(np.append(rng.uniform(0, 1, 3), 0.8).astype(np.float32))
        if i == bad:
            p["blend"] = 29
        more = {}
        if i % 9 < 4:
            cols = rng.uniform(0, 1, (2 + i % 3, 4)).astype(np.float32)
            p["gradient"] = b.add_gradient(1 + i % 4, (10.0, 20.0), (200.0, 120.0), (5.0, 90.0), cols)
        elif i % 9 == 4:
            more["image_shader"] = S.image_shader(img, tile_x=i % 4)
        if i % 7 == 2:
            more["color_filter"] = S.filter_record(S.FILTER_MATRIX, matrix=rng.uniform(-1, 1, 20))
        if i % 11 == 5:
            p["blur_style"], p["blur_radius"] = 1 + i % 4, float(rng.uniform(1, 6))
        if i % 97 == 40:
            b.save()
            b.clip_path(square, rng.uniform(0, 200, (4, 2)).astype(np.float32), S.CLIP_INTERSECT)
        b.draw_path(verbs, pts, p, **more)
        if i % 97 == 80:
            b.restore()
    return b.build().to_bytes()


def _compare(lib, bufs, threads):
    lib.skc_build_streams_compare.argtypes = [ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p,
                                              ctypes.c_uint]
    cbufs = [ctypes.create_string_buffer(b, len(b)) for b in bufs]
    ptrs = (ctypes.c_void_p * len(bufs))(*[ctypes.addressof(c) for c in cbufs])
    lens = (ctypes.c_size_t * len(bufs))(*[len(b) for b in bufs])
    return lib.skc_build_streams_compare(len(bufs), ptrs, lens, threads)


# 682 draws: one thread's share of 16384 verbs twice, less a draw; then two
# threads; then more draws than 16 threads take.  First canvas of a batch,
# and after another.
@pytest.mark.parametrize("draws,threads", [(682, 2), (683, 2), (1400, 3), (5700, 16)])
def test_threaded_draws_match_one_thread(cpu_pipeline, draws, threads):
    large = _one_large(draws)
    assert _compare(cpu_pipeline, [large], threads) == 0
    assert _compare(cpu_pipeline, [_streams()[8], large, large], threads) == 0


@pytest.mark.parametrize("bad", [0, 700, 1399])
def test_threaded_draws_report_a_bad_draw(cpu_pipeline, bad):
    assert _compare(cpu_pipeline, [_one_large(1400, bad)], 4) == -2


def test_threaded_draws_truncated(cpu_pipeline):
    large = _one_large(1400)
    assert _compare(cpu_pipeline, [large[:len(large) // 2]], 4) == -2
