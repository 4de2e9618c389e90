"""Early Z of the visibility path, whose lists come in no particular order: a
triangle may only be dropped if none of its samples could win. A plane's slopes
are floored to whole depth units per sample, so samples far from the centre of a
triangle over 2,048 pixels across can lie below the header's minimum depth by
more than the margin in it."""
import numpy as np
import pytest

from conftest import pkg_mod
from helpers import PIPES, PIPE_SAMPLES, assert_same, gpu_render, oracle_render, pkg, vertices_for
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

W = H = 4095
TILE = 510 * 8      # tile (510, 510), both ways
STEP = 2.0 ** -24   # clip z of 128 depth units near -1


def _tri(corners, z, rgb):
    """One triangle from pixel corners and depths in steps of 128 units above clip z = -1 + 2^-11."""
    v = np.zeros((3, 8), np.float32)
    v[:, 0] = np.array([c[0] for c in corners]) * (2.0 / W) - 1.0
    v[:, 1] = np.array([c[1] for c in corners]) * (2.0 / H) - 1.0
    v[:, 2] = -1.0 + 2.0 ** -11 + np.asarray(z) * STEP
    v[:, 3] = 1.0
    v[:, 4:7] = rgb
    v[:, 7] = 1.0
    return v


def _slanted(z):
    """Half the viewport, slopes just below -1 unit per pixel both ways: -2 once floored, so samples at its far
    corner lie some 4,000 units below the plane."""
    return _tri([(0.0, H), (W, 0.0), (W, H)], [z + 33, z + 33, z], (0.1, 0.9, 0.2))


def _scene(tris):
    v = np.concatenate(tris)
    return {"vertices": v, "indices": np.arange(v.shape[0], dtype=np.int32).reshape(-1, 3), "width": W, "height": H}


def _zmin(pipe, v):
    flags, blend, shader, stride = PIPES[pipe]
    op = orc.make_pipe(W, H, PIPE_SAMPLES.get(pipe, 1), flags, blend, shader, stride)
    _, hdr, data, _ = orc.setup(op, vertices_for(pipe, v), np.arange(3, dtype=np.int32).reshape(1, 3))
    d = data[0].astype(np.uint64)
    s = PIPE_SAMPLES.get(pipe, 1).bit_length() - 1
    corner = int((((d[0] * (TILE + 7) + d[1] * (TILE + 7)) << np.uint64(s)) + d[2]) & np.uint64(0xFFFFFFFF))
    return int(hdr[0, 3]) & ~0xFFF, corner


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_gouraud_flat"])
def test_samples_below_the_header_minimum_win(cuda, pipe):
    # A depth at which the header's minimum loses little to its rounding down to 4,096 units.
    z0 = next(z for z in range(200, 264) if _zmin(pipe, _slanted(z))[0] - _zmin(pipe, _slanted(z))[1] > 1024)
    zmin, corner = _zmin(pipe, _slanted(z0))
    # 64 layers over the tile, nearest first, deeper than the slanted triangle's samples there and nearer than its
    # header's minimum; small triangles come first in a tile's list.
    tris, x0, x1 = [], TILE, TILE + 8.0
    for k in range(64):
        for c in ([(x0, x0), (x1, x0), (x0, x1)], [(x1, x1), (x0, x1), (x1, x0)]):
            tris.append(_tri(c, [0, 0, 0], (0.9, 0.1, 0.1)))
    for lift in range(-64, 4096):   # the layers' depth, in steps
        if corner + 256 < _zmin(pipe, _tri([(x0, x0), (x1, x0), (x0, x1)], [lift] * 3, (0, 0, 0)))[1] < zmin - 256:
            break
    else:
        pytest.fail("no depth between the samples and the header's minimum")
    for t in tris:
        t[:, 2] += np.float32(lift * STEP)
    sc = _scene(tris + [_slanted(z0)])
    p = pkg()
    clear = (p.color_to_abgr(0.1, 0.2, 0.3, 1.0), p.clear_depth_from_float(1.0))
    rc, rd, st = oracle_render(pipe, sc, clear)
    assert st["zmin_violations"] > 0
    assert (rc[TILE:TILE + 8, TILE:TILE + 8] == rc[H - 100, W - 100]).any(), "the slanted triangle shows in the tile"
    for _ in range(2):
        c, d, cnt, _ = gpu_render(pipe, sc, clear)
        assert cnt["overflow"] == 0
        assert_same(c, d, rc, rd, f"{pipe} beyond 2,048 pixels")
