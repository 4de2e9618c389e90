"""Forms of the fine stage that depend on a triangle's extent or a surface's
address: triangles around 2,048 pixels across (32,767 subpixels is the most
that a packed record's edge steps hold), beyond 1,024 pixels from the tile
(the bound of the 32-bit edge values), every width of a small triangle's pixel
box, and surfaces that are only 4-byte aligned (moved word by word) with empty
and covered tiles, cleared and loaded. Exact, against the oracle."""
import numpy as np
import pytest
import torch

from helpers import PIPE_SAMPLES, assert_same, gpu_render, init_surfaces, oracle_render, pkg

pytestmark = pytest.mark.gpu

PIPES = ["PixelPipe_gouraud", "PixelPipe_gouraud_msaa2", "PixelPipe_gouraud_msaa4", "PixelPipe_gouraud_msaa8",
         "PixelPipe_gouraud_srcover", "PixelPipe_gouraud_nodepth", "PixelPipe_gouraud_srcover_msaa4",
         "PixelPipe_deriv_quads"]


def _scene(px, width, height, seed):
    """Triangles given as pixel positions [n, 3, 2], w = 1, random depth per vertex, colour and alpha."""
    rng = np.random.default_rng(seed)
    n = px.shape[0]
    v = np.empty((n, 3, 8), np.float32)
    v[..., 0] = px[..., 0] * (2.0 / width) - 1.0
    v[..., 1] = px[..., 1] * (2.0 / height) - 1.0
    v[..., 2] = rng.uniform(-0.9, 0.9, (n, 3))
    v[..., 3] = 1.0
    v[..., 4:7] = rng.integers(0, 256, (n, 3, 3)) / np.float32(255.0)
    v[..., 7] = rng.integers(40, 200, (n, 1)) / np.float32(255.0)
    return {"vertices": v.reshape(-1, 8), "indices": np.arange(3 * n, dtype=np.int32).reshape(-1, 3), "width": width,
            "height": height}


def _check(pipe, sc, what, cleared=True, **kw):
    p = pkg()
    clear = (p.color_to_abgr(0.1, 0.2, 0.3, 1.0), p.clear_depth_from_float(1.0)) if cleared else None
    color, depth = (None, None) if cleared else init_surfaces(sc, PIPE_SAMPLES.get(pipe, 1), 3)
    c, d, cnt, _ = gpu_render(pipe, sc, clear, color, depth, **kw)
    rc, rd, st = oracle_render(pipe, sc, clear, color, depth)
    assert cnt["overflow"] == 0 and st["zmin_violations"] == 0
    assert_same(c, d, rc, rd, what)


def _wide(width, height, seed):
    """Triangles of given extents on the longer axis, both windings, beside small ones."""
    rng = np.random.default_rng(seed)
    spans = np.array([2, 40, 1000, 1023, 1024, 1025, 2040, 2047, 2047.9375, 2048, 2048.0625, 2049, 3000, 4000.0])
    spans = np.repeat(spans, 4)[:, None]
    x0 = rng.uniform(0, 1, spans.shape) * np.maximum(4090 - spans, 0)
    x = np.concatenate([x0, x0 + spans, x0 + spans * rng.uniform(0, 1, spans.shape)], axis=1)
    y = rng.uniform(0, 200, x.shape)
    tri = np.stack([x, y], axis=-1)
    small = np.array([[0, 0], [5, 1], [1, 6]]) + rng.uniform(0, 1, (400, 1, 2)) * [4000, 190]
    tri = np.concatenate([tri, tri[:, ::-1], small, small[:, ::-1]])
    tri = tri[rng.permutation(tri.shape[0])]
    return _scene(tri if width > height else np.ascontiguousarray(tri[..., ::-1]), width, height, seed)


@pytest.mark.parametrize("pipe", PIPES)
@pytest.mark.parametrize("size", [(4095, 200), (200, 4095)])
def test_triangles_around_the_packed_extent(cuda, pipe, size):
    _check(pipe, _wide(*size, 11), f"{pipe} {size}")


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_gouraud_msaa4", "PixelPipe_gouraud_srcover"])
def test_every_box_width(cuda, pipe):
    """Boxes of 1 to 8 pixels each way, all dealt as pairs."""
    rng = np.random.default_rng(2)
    ext = np.stack(np.meshgrid(np.arange(1, 10), np.arange(1, 10)), axis=-1).reshape(-1, 1, 2).repeat(6, axis=0)
    unit = np.array([[0, 0], [1, 0.1], [0.1, 1.0]])
    tri = unit * ext + rng.uniform(0, 90, (ext.shape[0], 1, 2))
    tri = np.concatenate([tri, tri[:, ::-1]])
    _check(pipe, _scene(tri, 101, 99, 4), pipe, tuning=dict(fine_self_pixels=64))


@pytest.mark.parametrize("pipe", PIPES)
@pytest.mark.parametrize("cleared", [True, False])
@pytest.mark.parametrize("offsets", [(1, 0), (0, 1), (2, 2)])
def test_surface_addresses(cuda, monkeypatch, pipe, cleared, offsets):
    """Colour or depth 4 bytes off an 8-byte boundary, and both on one that is no multiple of 16."""
    p = pkg()
    base = p.CudaSurface

    class Offset(base):
        def __init__(self, size, fmt, numSamples=1, device="cuda"):
            super().__init__(size, fmt, numSamples, device)
            shift = offsets[0] if fmt == base.FORMAT_RGBA8 else offsets[1]
            n = self.tensor.numel()
            self.tensor = torch.zeros(n + 4, dtype=torch.int32, device=device)[shift:shift + n].view(self.tensor.shape)
            assert self.tensor.data_ptr() % 16 == 4 * shift

    monkeypatch.setattr(p, "CudaSurface", Offset)
    rng = np.random.default_rng(6)
    tri = np.array([[0, 0], [9, 1], [1, 12]]) + rng.uniform(0, 60, (150, 1, 2))   # the rest of the tiles stays empty
    _check(pipe, _scene(np.concatenate([tri, tri[:, ::-1]]), 150, 85, 7), f"{pipe} {offsets}", cleared)
