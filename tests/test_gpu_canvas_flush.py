"""A canvas flushed again and again with different draws each time: every
flush renders its own draws over the pixels of the flushes before it.
Against the oracle's render of all draws in one scene."""
import numpy as np
import pytest

from skity_gb300 import scene as S
from skity_gb300.canvas import Canvas, Paint, Path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1, 5, 2), (7, 1, 9), (3, 3, 3)])
def test_each_flush_renders_its_own_draws(gpu_ctx, oracle_lib, counts):
    rng = np.random.default_rng(sum(counts))
    bitmap = np.zeros((48, 60, 4), np.uint8)
    canvas = Canvas.MakeCUDACanvas(gpu_ctx, bitmap)
    canvas.Clear((0.0, 0.5, 1.0, 1.0))
    sb = S.SceneBuilder(60, 48, clear=(0.0, 0.5, 1.0, 1.0))
    for n in counts:
        for _ in range(n):
            k = int(rng.integers(3, 9))
            pts = rng.uniform(0, 60, (k, 2)).astype(np.float32)
            color = tuple(float(v) for v in rng.uniform(0.2, 1.0, 4).astype(np.float32))
            path = Path().MoveTo(*pts[0])
            for q in pts[1:]:
                path.LineTo(*q)
            canvas.DrawPath(path.Close(), Paint().SetFillColor(*color))
            p = S.default_paint()
            p["fill_color"] = color
            sb.draw_path(path.verbs, pts, p)
        canvas.Flush()
    assert oracle_lib.compare(bitmap, oracle_lib.render(sb.build())[0])["bad_pixels"] == 0
