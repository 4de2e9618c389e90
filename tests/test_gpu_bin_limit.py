"""Bin entries are counted, not stored: a draw with more of them than the
estimate of two a triangle is drawn at once -- blocking without a rerun, queued
and static without being skipped or refused -- while a limit set by the caller
holds."""
import numpy as np
import pytest
import torch

from helpers import assert_same, gpu_render, oracle_render, pkg
from test_gpu_tile_lists import _clear, _triangles
from test_zz_no_alloc import _draw_static, _static_fn

pytestmark = pytest.mark.gpu

SIZE = 1024


def _corner_scene(n, large, seed):
    """n triangles each over the corner of four bins (of 128 pixels), and `large` ones over 5x5 bins."""
    rng = np.random.default_rng(seed)
    corner = 128.0 * rng.integers(1, 8, (n, 1, 2))
    tri = corner + np.array([[-5.0, -5.0], [6.0, -4.0], [-4.0, 6.0]]) + rng.uniform(-0.5, 0.5, (n, 3, 2))
    big = 128.0 * rng.integers(0, 4, (large, 1, 2)) + np.array([[10.0, 10.0], [600.0, 20.0], [20.0, 600.0]])
    return _triangles(np.concatenate([tri, big]), SIZE, SIZE, seed)


def _queued(cr, sc):
    p = pkg()
    s = [p.CudaSurface((SIZE, SIZE), f, 1) for f in (p.CudaSurface.FORMAT_RGBA8, p.CudaSurface.FORMAT_DEPTH32)]
    cr.setSurfaces(*s)
    cr.setPixelPipe(None, "PixelPipe_gouraud")
    v, i = torch.from_numpy(sc["vertices"]).cuda(), torch.from_numpy(sc["indices"]).cuda()
    cr.setVertexBuffer(v, 0)
    cr.setIndexBuffer(i, 0, i.shape[0])
    cr._check(cr._lib.cr_deferred_clear_raw(cr._ctx, *_clear()))
    cr.drawTrianglesAsync()
    torch.cuda.synchronize()
    return (*(t.download().numpy().astype(np.uint32) for t in s), cr.getCounters())


def test_more_bin_entries_than_the_estimate(cuda):
    n = 100000
    sc = _corner_scene(n, 0, 1)
    rc, rd, _ = oracle_render("PixelPipe_gouraud", sc, _clear())
    c, d, cnt, _ = gpu_render("PixelPipe_gouraud", sc, _clear())
    assert cnt["bin_entries"] == 4 * n > 2 * n + 65536
    assert cnt["reruns"] == 0 and cnt["overflow"] == 0
    assert_same(c, d, rc, rd, "blocking draw")
    cr = pkg().CudaRaster()
    cr.init()
    c, d, cnt = _queued(cr, sc)
    assert cnt["overflow"] == 0
    assert_same(c, d, rc, rd, "queued draw of a fresh context")


def test_limit_of_the_caller_holds(cuda):
    sc = _corner_scene(1000, 0, 2)
    cr = pkg().CudaRaster()
    cr.init()
    cr.setCapacity(1000, 3999, 100000)
    c, d, cnt = _queued(cr, sc)
    assert cnt["overflow"] != 0 and cnt["bin_entries"] == 4000
    assert (c == 0).all() and (d == 0).all(), "a skipped draw changed the surfaces"
    cr.setCapacity(1000, 4000, 100000)
    c, d, cnt = _queued(cr, sc)
    rc, rd, _ = oracle_render("PixelPipe_gouraud", sc, _clear())
    assert cnt["overflow"] == 0
    assert_same(c, d, rc, rd, "limit met")


def test_static_draw_with_many_bin_entries(cuda):
    sc = _corner_scene(65500, 36, 3)
    rc, rd, _ = oracle_render("PixelPipe_gouraud", sc, _clear())
    _, _, cnt, _ = gpu_render("PixelPipe_gouraud", sc, _clear())
    assert cnt["bin_entries"] > 4 * 65536
    c, d, _ = _draw_static(_static_fn(), "PixelPipe_gouraud", sc, _clear(), cuda)
    assert_same(c, d, rc, rd, "static draw")
