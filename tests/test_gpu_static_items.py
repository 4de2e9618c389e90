"""The static draw close to its tile queue (1,048,576 entries) with all entries
from items, spread over every warp of the item kernel: each leaves a block of
records partly filled, and all must have room. Against the oracle, exact."""
import numpy as np
import pytest

from helpers import assert_same, gpu_render, oracle_render
from test_gpu_tile_lists import _clear, _triangles
from test_zz_no_alloc import _draw_static, _static_fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_gouraud_srcover"])
@pytest.mark.parametrize("kind", ["huge", "medium"])
def test_static_draw_full_of_items(cuda, pipe, kind):
    rng = np.random.default_rng(4)
    if kind == "huge":   # half the viewport each
        corners = np.array([[1.0, 1.0], [1023.0, 1.0], [1.0, 1023.0], [1023.0, 1023.0]])
        tri = corners[np.array([[0, 1, 2], [3, 2, 1]])][np.arange(124) % 2]
    else:                # 3x3 to 5x5 tiles
        tri = rng.uniform(30, 994, (60000, 1, 2)) + np.array([[-15.0, -15.0], [15.0, -14.0], [-14.0, 15.0]]) \
            * rng.uniform(0.7, 1.0, (60000, 1, 1))
    sc = _triangles(tri, 1024, 1024, 5)
    rc, rd, _ = oracle_render(pipe, sc, _clear())
    _, _, cnt, _ = gpu_render(pipe, sc, _clear())
    assert (2**20 - 2**17 if kind == "huge" else 2**19) < cnt["tile_entries"] <= 2**20
    fn = _static_fn()
    for call in range(2):
        c, d, _ = _draw_static(fn, pipe, sc, _clear(), cuda)
        assert_same(c, d, rc, rd, f"{pipe} {kind} static call {call}")
