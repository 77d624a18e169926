"""The register sweeps where their sizes change: combs of slanted teeth whose
active list sits at and around 32, 64 and 128 edges (the forms' limits) and
past them, in rows wider than the on-chip accumulator (3,072 pixels), with
shallow teeth (long partial rows: more accumulator entries than one flush
gathers) and curved ones (a piece change every few rows).  Against the oracle."""
import numpy as np
import pytest

from skity_gb300 import scene as S

pytestmark = pytest.mark.gpu


def comb_scene(teeth, width, height, slant, curved, evenodd):
    """`teeth` triangles side by side over the whole canvas, each crossed by
    its neighbours when the slant is large."""
    rng = np.random.default_rng(1000 * teeth + width + int(curved))
    b = S.SceneBuilder(width, height)
    verbs, pts = [S.MOVE], [(0.3, height - 0.7)]
    step = (width - 1.0) / teeth
    for i in range(teeth):
        x = 0.3 + i * step
        top = (x + step * (0.5 + slant), float(rng.uniform(0.1, 0.3) * height))
        end = (x + step, height - float(rng.uniform(0.2, 2.0)))
        if curved:
            verbs += [S.QUAD, S.QUAD]
            pts += [(x + step * slant, 0.6 * height), top, (x + step, 0.5 * height), end]
        else:
            verbs += [S.LINE, S.LINE]
            pts += [top, end]
    verbs.append(S.CLOSE)
    p = S.default_paint()
    p["fill_type"] = S.EVEN_ODD if evenodd else S.WINDING
    p["fill_color"] = (0.2, 0.5, 0.9, 0.7)
    b.draw_path(verbs, pts, p)
    return b.build()


@pytest.mark.parametrize("teeth,width,height,slant,curved", [
    (15, 61, 40, 0.1, False), (16, 64, 40, 0.1, True), (17, 333, 40, 2.5, False),
    (31, 129, 48, 0.2, True), (32, 640, 48, 3.0, False), (33, 200, 24, 0.0, False),
    (63, 500, 32, 0.3, True), (64, 257, 32, 5.0, False), (65, 1000, 16, 0.1, True),
    (16, 3300, 9, 6.0, False), (40, 3300, 9, 20.0, False), (90, 700, 20, 8.0, True)])
def test_forms_match_oracle(gpu_ctx, oracle_lib, teeth, width, height, slant, curved):
    scenes = [comb_scene(teeth, width, height, slant, curved, e) for e in (False, True)]
    for sc, got in zip(scenes, gpu_ctx.render_streams(scenes)):
        assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0


@pytest.mark.parametrize("teeth,slant,curved", [(12, 0.2, True), (17, 1.5, False), (33, 2.0, True),
                                                (70, 4.0, False)])
def test_forms_under_path_clips(gpu_ctx, oracle_lib, teeth, slant, curved):
    """Passes that keep raw spans (clip paths and the draws under them) in each
    form: a comb drawn under a comb."""
    width, height = 300, 30
    comb = comb_scene(teeth, width, height, slant, curved, True)
    scenes = []
    # a difference sorts each row: 256 spans at most, fewer than 70 teeth make
    for op in (S.CLIP_INTERSECT, S.CLIP_DIFFERENCE) if teeth < 70 else (S.CLIP_INTERSECT,):
        b = S.SceneBuilder(width, height)
        b.clip_path(comb.verbs, comb.points + np.float32(0.37), op, S.EVEN_ODD)
        p = S.default_paint()
        p["fill_color"] = (0.7, 0.2, 0.3, 0.8)
        b.draw_path(comb.verbs, comb.points, p)
        scenes.append(b.build())
    for sc, got in zip(scenes, gpu_ctx.render_streams(scenes)):
        assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0


# at most 256 active edges: two a tooth, and what a slant adds
@pytest.mark.parametrize("teeth,width,height,slant,curved",
                         [(65, 513, 24, 0.0, False), (100, 400, 24, 0.4, True),
                          (127, 700, 20, 0.1, False), (128, 1024, 17, 0.0, True),
                          (129, 1024, 17, 0.0, False), (150, 3300, 9, 6.0, True),
                          (300, 900, 12, 3.0, False)])
@pytest.mark.parametrize("evenodd", [False, True])
def test_long_lists_match_oracle(gpu_ctx, oracle_lib, teeth, width, height, slant, curved, evenodd):
    sc = comb_scene(teeth, width, height, slant, curved, evenodd)
    got = gpu_ctx.render_streams([sc])[0]
    assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0
