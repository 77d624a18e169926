"""skity_cuda_draw_path_static takes nothing from the host heap, whatever the
path's size (tests/static_heap.cc counts), and draws what render_streams
draws.  Sizes: the smallest path; 1,344 points, the longest path of 12 KiB
(copied together with the draw's descriptors), and one more (copied from the
caller's memory); one of 180 KB.  Conic weights on either side too."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, TESTS
from skity_gb300 import build
from skity_gb300 import scene as S

pytestmark = pytest.mark.gpu


def test_no_host_heap(gpu_ctx):
    out = os.path.join(TESTS, "_build", "static_heap")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    r = subprocess.run([build.nvcc(), "-std=c++17", "-O2", "-I" + os.path.join(ROOT, "include"),
                        os.path.join(TESTS, "static_heap.cc"), "-o", out, "-L" + build.BUILD,
                        "-lskity_cuda", "-Xlinker", "-rpath=" + build.BUILD,
                        "-Xlinker", "--export-dynamic"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    sizes = ["3", "1344", "1345", "20000"]
    r = subprocess.run([out, *sizes], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split("\n")[:-1] == [f"{n} 0 0" for n in sizes]


@pytest.mark.parametrize("n,conics", [(3, 0), (1344, 0), (1345, 0), (20000, 0), (1100, 300),
                                      (1300, 300)])
def test_draws_what_render_streams_draws(gpu_ctx, n, conics):
    import torch
    from test_zz_no_alloc import _static_draw, _white_canvas
    from skity_gb300 import _lib
    b = S.SceneBuilder(256, 200)
    t = np.linspace(0, 2 * np.pi, n, endpoint=False)
    pts = np.stack([128 + (40 + np.arange(n) % 50) * np.cos(t),
                    100 + (40 + np.arange(n) % 50) * np.sin(t)], 1).astype(np.float32)
    # MoveTo, `conics` of two points each, lines
    verbs = [S.MOVE] + [S.CONIC] * conics + [S.LINE] * (n - 1 - 2 * conics)
    p = S.default_paint()
    p["fill_color"] = (0.7, 0.2, 0.4, 0.6)
    b.draw_path(verbs, pts, p, weights=[0.5 + 0.01 * (i % 90) for i in range(conics)])
    sc = b.build()
    canvas = _white_canvas(torch, 200, 256)
    assert _static_draw(_lib.load(), canvas, sc, 0, torch.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(canvas.cpu().numpy(), gpu_ctx.render_streams([sc])[0])
