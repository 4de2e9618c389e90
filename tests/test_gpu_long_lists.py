"""Tile lists beyond the shared-memory sort (4,096 entries), which a CTA sorts
by radix passes of 8 bits through a copy: two, three and four passes, lengths
around a warp's and the CTA's pieces, several long lists at once, subtriangles
of clipped triangles among them, and the static draw, whose copy lies in its own
scratch. Blended framebuffers show any entry out of order; exact."""
import numpy as np
import pytest

from helpers import assert_same, gpu_render, oracle_render
from test_gpu_tile_lists import _check, _clear, _triangles
from test_zz_no_alloc import _draw_static, _static_fn

pytestmark = pytest.mark.gpu


def _crowd(n, seed, size=8):
    rng = np.random.default_rng(seed)
    return np.array([[0.5, 0.5], [size - 0.5, 0.5], [0.5, size - 0.5]]) + rng.uniform(-0.4, 0.4, (n, 3, 2))


@pytest.mark.parametrize("n", [4097, 4351, 4353, 8192, 8193, 8449, 30011])
def test_one_long_list(cuda, n):
    """Up to 8,192 triangles: 16-bit entries, two passes; beyond: three, the result copied back."""
    cnt = _check("PixelPipe_gouraud_nodepth", _triangles(_crowd(n, n), 16, 16, n), f"{n} triangles in one tile")
    assert cnt["tile_entries"] >= n


def test_four_passes(cuda):
    """Over 2^21 triangles (25-bit entries), all but 6,000 without area."""
    n = 2100000
    rng = np.random.default_rng(3)
    tri = np.full((n, 3, 2), 4.0)
    tri[np.sort(rng.choice(n, 6000, replace=False))] = _crowd(6000, 4)
    cnt = _check("PixelPipe_gouraud_nodepth", _triangles(tri, 16, 16, 5), "four passes")
    assert cnt["tile_entries"] >= 6000


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud_srcover", "PixelPipe_trihash_srcover"])
def test_many_long_lists_with_clipped_triangles(cuda, pipe):
    """32 tiles with lists of a few entries to 9,000, many of them of several subtriangles."""
    rng = np.random.default_rng(9)
    at = rng.integers(0, 3, (9000, 1, 2)) * rng.integers(0, 2, (9000, 1, 2)) * 8.0
    sc = _triangles(_crowd(9000, 10) + at, 64, 32, 11)
    v = sc["vertices"].reshape(-1, 3, 8)
    v[::5, 0, 2] = -1.5      # through the near plane
    v[2::25, 1, 2] = 1.25    # and the far one
    sc["vertices"] = v.reshape(-1, 8)
    cnt = _check(pipe, sc, f"{pipe} long lists")
    assert cnt["num_subtris"] > cnt["num_tris"] and cnt["tile_entries"] > 9000


def test_static_draw_with_long_lists(cuda):
    sc = _triangles(_crowd(20000, 12, 14), 24, 24, 13)
    rc, rd, _ = oracle_render("PixelPipe_gouraud_nodepth", sc, _clear())
    fn = _static_fn()
    for _ in range(2):
        c, d, _ = _draw_static(fn, "PixelPipe_gouraud_nodepth", sc, _clear(), cuda)
        assert_same(c, d, rc, rd, "static draw with long lists")
    c, d, cnt, _ = gpu_render("PixelPipe_gouraud_nodepth", sc, _clear())
    assert cnt["tile_entries"] > 4 * 4096
    assert_same(c, d, rc, rd, "context draw with long lists")
