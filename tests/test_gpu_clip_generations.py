"""Path clips by generation: chains of clips one inside another, siblings under
one parent, and clips off the canvas in the middle of a chain (no rows of their
own), in one canvas and over several.  Against the oracle."""
import numpy as np
import pytest

from skity_gb300 import scene as S

pytestmark = pytest.mark.gpu


def tree_scene(seed, groups, depth, off_at, op):
    rng = np.random.default_rng(seed)
    b = S.SceneBuilder(70, 50)
    quad = [S.MOVE, S.LINE, S.QUAD, S.CLOSE]

    def draw():
        p = S.default_paint()
        p["fill_color"] = tuple(rng.uniform(0.2, 0.9, 4).astype(np.float32))
        b.draw_path(quad, rng.uniform(-5, 75, (4, 2)).astype(np.float32), p)

    for _ in range(groups):
        b.save()
        for d in range(depth):
            pts = rng.uniform(-20, 90, (4, 2)).astype(np.float32)
            if d == off_at:
                pts += np.float32(500)
            b.clip_path(quad, pts, op if d % 2 else S.CLIP_INTERSECT)
            draw()
            b.save()  # a sibling of the next clip
            b.clip_path(quad, rng.uniform(0, 60, (4, 2)).astype(np.float32), op)
            draw()
            b.restore()
        b.restore()
        draw()
    return b.build()


@pytest.mark.parametrize("groups,depth,off_at", [(1, 1, -1), (1, 6, -1), (5, 3, 1), (9, 2, 0), (2, 4, 3)])
def test_generations_match_oracle(gpu_ctx, oracle_lib, groups, depth, off_at):
    scenes = [tree_scene(10 * groups + depth, groups, depth, off_at, op)
              for op in (S.CLIP_INTERSECT, S.CLIP_DIFFERENCE)]
    for sc, got in zip(scenes, gpu_ctx.render_streams(scenes)):
        assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0
