"""Gradient canvases whose width is not a multiple of 4: the compositor keeps
each row tile in shared memory with the gradient's stops behind it, and the
stop colours are read 16 bytes at a time.  Each canvas against the oracle."""
import pytest

from skity_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [33, 34, 35, 129, 390, 1023])
def test_gradients_at_any_width(gpu_ctx, oracle_lib, width):
    sc = S.random_paths_scene(S.SEED_BASE + 600 + width, width, 41, 24, 3, 12, gradient_frac=0.8,
                              evenodd_frac=0.3, stroke_frac=0.2)
    got = gpu_ctx.render_streams([sc])[0]
    assert oracle_lib.compare(got, oracle_lib.render(sc)[0])["bad_pixels"] == 0
