"""The tile lists at the sizes where building them changes course: list lengths
around the sort's limits (8, 16 and 32 lanes, register runs, shared memory,
global merges), boxes of at most 2x2 tiles that fill a chunk's pair room,
boxes around the medium / large / huge limits, and batches with more bins and
tiles than the spread counters take. Framebuffers of blending pipes show any
list out of submission order or with a missing entry; all comparisons are
exact."""
import numpy as np
import pytest
import torch

from conftest import pkg_mod
from helpers import assert_same, gpu_render, oracle_render, pkg

pytestmark = pytest.mark.gpu


def _clear():
    p = pkg()
    return p.color_to_abgr(0.1, 0.2, 0.3, 1.0), p.clear_depth_from_float(1.0)


def _triangles(px, width, height, seed):
    """Scene of triangles given as pixel positions [n, 3, 2], w = 1, random depth, colour and alpha."""
    rng = np.random.default_rng(seed)
    n = px.shape[0]
    v = np.empty((n, 3, 8), np.float32)
    v[..., 0] = px[..., 0] * (2.0 / width) - 1.0
    v[..., 1] = px[..., 1] * (2.0 / height) - 1.0
    v[..., 2] = rng.uniform(-0.9, 0.9, (n, 1))
    v[..., 3] = 1.0
    v[..., 4:7] = rng.integers(0, 256, (n, 1, 3)) / np.float32(255.0)
    v[..., 7] = rng.integers(40, 200, (n, 1)) / np.float32(255.0)
    return {"vertices": v.reshape(-1, 8), "indices": np.arange(3 * n, dtype=np.int32).reshape(-1, 3), "width": width,
            "height": height}


def _check(pipe, sc, what, **kw):
    c, d, cnt, _ = gpu_render(pipe, sc, _clear(), **kw)
    rc, rd, st = oracle_render(pipe, sc, _clear())
    assert cnt["overflow"] == 0 and st["zmin_violations"] == 0
    assert_same(c, d, rc, rd, what)
    return cnt


@pytest.mark.parametrize("n", [1, 2, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 255, 256, 257, 512, 513, 1025, 4096, 4097,
                               8193, 9001])
def test_blended_list_lengths(cuda, n):
    """n triangles over one crowded tile of a small viewport (dense lists)."""
    rng = np.random.default_rng(n)
    tri = np.array([[0.5, 0.5], [7.5, 0.5], [0.5, 7.5]]) + rng.uniform(-0.4, 0.4, (n, 3, 2))
    cnt = _check("PixelPipe_gouraud_nodepth", _triangles(tri, 16, 16, n), f"{n} triangles in one tile")
    assert cnt["tile_entries"] >= n


def test_blended_sparse_lists_beside_crowded_tiles(cuda):
    """Mostly short lists (four tiles a warp) with tiles of 12, 40, 300 and 5000 entries among them."""
    rng = np.random.default_rng(5)
    sc = [np.array([[0, 0], [5, 1], [1, 5]]) + rng.uniform(0, 505, (20000, 1, 2))]
    for n, x, y in ((12, 40, 40), (40, 200, 8), (300, 8, 300), (5000, 400, 400)):
        sc.append(np.array([[x + 0.5, y + 0.5], [x + 7.4, y + 0.5], [x + 0.5, y + 7.4]]) + rng.uniform(-0.3, 0.3, (n, 3, 2)))
    tri = rng.permutation(np.concatenate(sc))
    cnt = _check("PixelPipe_trihash_srcover", _triangles(tri, 512, 512, 6), "sparse lists beside crowded tiles")
    assert cnt["tile_entries"] < 16 * cnt["num_tiles"]


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_gouraud_srcover", "PixelPipe_gouraud_msaa8"])
@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 1000])
def test_four_tiles_per_triangle_fill_the_pair_room(cuda, pipe, n):
    """Every triangle in exactly 2x2 tiles: twice the pair records a chunk has room for."""
    rng = np.random.default_rng(n)
    corner = 8.0 * rng.integers(1, 12, (n, 1, 2))
    tri = corner + np.array([[-5.0, -5.0], [6.0, -4.0], [-4.0, 6.0]]) + rng.uniform(-0.5, 0.5, (n, 3, 2))
    cnt = _check(pipe, _triangles(tri, 101, 99, n), f"{pipe} {n} triangles over tile corners")
    assert cnt["tile_entries"] == 4 * n


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_gouraud_srcover"])
def test_boxes_around_the_item_limits(cuda, pipe):
    """Boxes of 2x2, 3x1, 1x3, 8x8, 8x9, 32x32, 32x33 and all tiles, thin and full, mixed with small ones."""
    rng = np.random.default_rng(8)
    parts = [rng.uniform(0, 500, (400, 1, 2)) + rng.uniform(-6, 6, (400, 3, 2))]
    for w, h in ((2, 2), (3, 1), (1, 3), (8, 8), (8, 9), (9, 8), (32, 32), (32, 33), (64, 50), (1, 50), (64, 1)):
        for k in range(6):
            x0 = 8 * rng.integers(0, 64 - w + 1) + 1.0
            y0 = 8 * rng.integers(0, 50 - h + 1) + 1.0
            x1, y1 = x0 + 8 * w - 2.0, y0 + 8 * h - 2.0
            full = [[x0, y0], [x1, y0], [x0, y1]] if k % 2 else [[x1, y1], [x0, y1], [x1, y0]]
            thin = [[x0, y0], [x1, y1], [x1 - 1.0, y1]]
            parts.append(np.array([full if k < 4 else thin]))
    tri = rng.permutation(np.concatenate(parts))
    _check(pipe, _triangles(tri, 512, 400, 9), f"{pipe} item limits")


def test_batch_beyond_the_shared_bins_and_spread_tiles(cuda):
    """17 scenes of 2048x2048: 4,352 bins and 1.1M tiles; each equals its single draw."""
    p = pkg()
    scenes = pkg_mod("scenes")
    items, insts = [], []
    for k in range(17):
        pipe = "PixelPipe_gouraud_srcover" if k % 2 else "PixelPipe_gouraud"
        sc = scenes.soup(3000 + 101 * k, 2048, 2048, seed=50 + k, median_px=12.0, alpha_range=(0.2, 1.0))
        cs = p.CudaSurface((2048, 2048), p.CudaSurface.FORMAT_RGBA8, 1)
        ds = p.CudaSurface((2048, 2048), p.CudaSurface.FORMAT_DEPTH32, 1)
        items.append((pipe, sc))
        insts.append({"pipe": pipe, "color": cs, "depth": ds, "vertices": torch.from_numpy(sc["vertices"]).cuda(),
                      "indices": torch.from_numpy(sc["indices"]).cuda(), "numTris": sc["indices"].shape[0],
                      "clear": (0.1, 0.2, 0.3, 1.0, 1.0)})
    cr = p.CudaRaster()
    cr.init()
    cr.drawBatch(insts)
    torch.cuda.synchronize()
    cnt = cr.getCounters()
    assert cnt["num_bins"] > 2048 and cnt["num_tiles"] > 1 << 20
    for (pipe, sc), it in zip(items, insts):
        c, d, _, _ = gpu_render(pipe, sc, _clear())
        assert_same(it["color"].download().numpy().astype(np.uint32), it["depth"].download().numpy().astype(np.uint32),
                    c, d, f"batched {pipe} {sc['indices'].shape[0]}")
