"""Compositor batches at their edges: spans of 1 to 70 pixels and spans across
the 1,024-pixel row tiles, side by side and overlapping, in solid, gradient and
other (kSrc) paints, on canvases narrower and wider than a tile.  Against the
oracle."""
import numpy as np
import pytest

from skity_gb300 import scene as S

pytestmark = pytest.mark.gpu


def bars_scene(width, kind):
    """One path of many bars per draw: pixel-aligned and slanted, so a row has
    runs of every length between their antialiased ends."""
    rng = np.random.default_rng(width + 7 * kind)
    b = S.SceneBuilder(width, 12)
    for d in range(6):
        verbs, pts, x = [], [], 0.0
        while x < width and len(pts) < 400:
            w = float(rng.integers(1, 71)) if d < 5 else float(width)
            slant = 0.0 if d % 2 else float(rng.uniform(-3, 3))
            verbs += [S.MOVE, S.LINE, S.LINE, S.LINE, S.CLOSE]
            pts += [(x, 0.25 * d), (x + w, 0.25 * d), (x + w + slant, 12), (x + slant, 12)]
            x += w + float(rng.integers(0, 4))
        p = S.default_paint()
        p["fill_color"] = tuple(rng.uniform(0.2, 0.9, 4).astype(np.float32))
        p["fill_type"] = d % 2
        if kind == 1:
            k = 2 + d
            cols = rng.uniform(0, 1, (k, 4)).astype(np.float32)
            offs = np.sort(rng.uniform(0, 1, k)).astype(np.float32)
            g = S.GRAD_RADIAL if d % 2 else S.GRAD_LINEAR
            p["gradient"] = b.add_gradient(g, (0.3 * width, 4.0), (0.6 * width, 9.0),
                                           (0.4 * width if d % 2 else 0.0, 0.0), cols, offs, d % 4)
        elif kind == 2:
            p["blend"] = S.BLEND_SRC
        b.draw_path(verbs, pts, p)
    return b.build()


@pytest.mark.parametrize("width", [31, 97, 1023, 1025, 2200])
def test_spans_match_oracle(gpu_ctx, oracle_lib, width):
    scenes = [bars_scene(width, k) for k in range(3)]
    for sc, got in zip(scenes, gpu_ctx.render_streams(scenes)):
        assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0


# The canvases above are the whole batch and take 64-pixel tiles; beside a
# filler of more work (60 draws on so many rows) theirs are wider, up to all of
# their 1,025 pixels
@pytest.mark.parametrize("rows", [4, 40, 400, 4000])
def test_tile_widths_match_oracle(gpu_ctx, oracle_lib, rows):
    b = S.SceneBuilder(900, rows)
    for k in range(60):
        p = S.default_paint()
        p["fill_color"] = (0.1, 0.2, 0.3, 0.5)
        b.draw_path([S.MOVE, S.LINE, S.LINE, S.LINE, S.CLOSE],
                    [(0, 0), (900 - k, 0.5), (900 - k, rows), (3.3 * k, rows)], p)
    scenes = [bars_scene(1025, k) for k in range(3)] + [b.build()]
    for sc, got in zip(scenes, gpu_ctx.render_streams(scenes)):
        assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0
