"""StackBlur at the edges of its kernels: strips of up to 372 rows and rows of up
to 6,144 words are staged in shared memory, larger ones are not; sums of lines
past 32,770 pixels at radius 254 need 64 bits.  Against the oracle."""
import numpy as np
import pytest

from skity_gb300 import scene as S

pytestmark = pytest.mark.gpu


def box_scene(w, h, radius, style):
    """A w x h pixel temp canvas: a box with a slanted side and the radius'
    margin around it, in two colours of unequal channels."""
    b = S.SceneBuilder(min(w, 700), min(h, 700))
    for k, color in enumerate([(0.9, 0.3, 0.1, 0.8), (0.1, 0.7, 0.4, 0.6)]):
        p = S.default_paint()
        p["fill_color"] = color
        p["blur_style"], p["blur_radius"] = style, float(radius)
        l, t, inner = -2.0 * k, -3.0 * k, h - 2 * radius
        if inner > 16384:  # as tall as coordinates go: centred, and not moved up
            t, inner = 3.0 * k - inner // 2, inner - 6 * k
        r, d = l + max(w - 2 * radius, 1), t + max(inner, 1)
        b.draw_path([S.MOVE, S.LINE, S.LINE, S.LINE, S.CLOSE],
                    [(l, t), (r, t), (r, d), (l + 0.3 * (r - l), d)], p)
    return b.build()


@pytest.mark.parametrize("w,h,radius,style",
                         [(1, 1, 1, 1), (5, 3, 2, 1), (33, 372, 7, 1), (31, 373, 7, 2),
                          (96, 600, 30, 1), (6143, 20, 5, 1), (6145, 20, 5, 3), (600, 520, 254, 1),
                          (515, 33276, 254, 1)])
def test_blur_matches_oracle(gpu_ctx, oracle_lib, w, h, radius, style):
    sc = box_scene(w, h, radius, style)
    got = gpu_ctx.render_streams([sc])[0]
    assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0
