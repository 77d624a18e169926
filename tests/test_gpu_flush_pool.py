"""A flush that blends over the bitmap's pixels and runs out of span pool: the
render is repeated with a larger pool, and every draw lands once.  A context
starts with a pool of 2^20 spans and a pass with spans takes 4,096 of them at
least, so 256 visible passes fit it and more do not.  Against the oracle's
render of all draws in one scene."""
import numpy as np
import pytest

from skity_gb300 import scene as S
from skity_gb300.canvas import Canvas, Context, MaskFilter, Paint, Path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("draws,blend,blur,short", [
    (256, 3, False, False), (257, 3, False, True), (300, 3, True, True),
    (600, 3, False, True), (300, 24, False, True)])  # 24: the general compositor
def test_every_draw_lands_once(gpu_ctx, oracle_lib, draws, blend, blur, short):
    rng = np.random.default_rng(draws)
    ctx = Context(0)
    bitmap = np.zeros((48, 60, 4), np.uint8)
    canvas = Canvas.MakeCUDACanvas(ctx, bitmap)
    canvas.Clear((0.0, 0.5, 1.0, 1.0))
    sb = S.SceneBuilder(60, 48, clear=(0.0, 0.5, 1.0, 1.0))

    def draw(filtered=False, mode=3):
        pts = (rng.uniform(12, 36, 2) + np.array([(0, -8), (-8, 7), (8, 7)]) +
               rng.uniform(-2, 2, (3, 2))).astype(np.float32)
        color = tuple(float(v) for v in rng.uniform(0.1, 0.5, 4).astype(np.float32))
        path = Path().MoveTo(*pts[0]).LineTo(*pts[1]).LineTo(*pts[2]).Close()
        paint = Paint().SetFillColor(*color).SetBlendMode(mode)
        p = S.default_paint()
        p["fill_color"], p["blend"] = color, mode
        if filtered:
            paint.SetMaskFilter(MaskFilter.MakeBlur(1, 2.0))
            p["blur_style"], p["blur_radius"] = 1, 2.0
        canvas.DrawPath(path, paint)
        sb.draw_path(path.verbs, pts, p)

    for _ in range(3):
        draw()
    canvas.Flush()
    for i in range(draws):
        draw(blur and i == 5, blend if i % 50 == 7 else 3)
    canvas.Flush()
    assert (ctx.stats()["retries"] > 0) == short
    assert oracle_lib.compare(bitmap, oracle_lib.render(sb.build())[0])["bad_pixels"] == 0
    canvas.close()
    ctx.close()


def test_empty_canvases_in_a_new_context(gpu_ctx):
    """A plan without passes falls short of nothing, in a context without a pool."""
    ctx = Context(0)
    scenes = [S.SceneBuilder(40 + i, 30, clear=(1.0, 0.5, 0.0, 1.0)).build() for i in range(3)]
    for _ in range(2):
        for sc, img in zip(scenes, ctx.render_streams(scenes)):
            assert img.shape == (30, sc.width, 4) and (img == img[0, 0]).all() and img[0, 0, 3] == 255
    ctx.close()
