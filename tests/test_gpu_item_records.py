"""Draws with more item pairs (tiles of boxes larger than 2x2) than a context
keeps records for (2^23): a blocking draw makes room and reruns, queued and
captured ones (and blocking ones beside a captured graph) find the pairs without
a record again. Opaque and blended, against the oracle, exact."""
import numpy as np
import pytest
import torch

from helpers import assert_same, gpu_render, oracle_render, pkg
from test_gpu_tile_lists import _clear, _triangles

pytestmark = pytest.mark.gpu

SIZE = 512
RECORDS = 1 << 23


def _scene(seed):
    """5,000 triangles of about half the viewport each (2,080 tiles) among small and medium ones."""
    rng = np.random.default_rng(seed)
    corners = np.array([[0.0, 0.0], [SIZE, 0.0], [0.0, SIZE], [SIZE, SIZE]])
    half = corners[np.array([[0, 1, 2], [3, 2, 1], [1, 3, 0], [2, 0, 3]])][np.arange(5000) % 4]
    half = np.clip(half + rng.uniform(-6.0, 6.0, half.shape), 0.0, SIZE)
    medium = rng.uniform(0, SIZE - 70, (3000, 1, 2)) + rng.uniform(0, 70, (3000, 3, 2))
    small = rng.uniform(0, SIZE - 9, (3000, 1, 2)) + rng.uniform(0, 9, (3000, 3, 2))
    return _triangles(rng.permutation(np.concatenate([half, medium, small])), SIZE, SIZE, seed)


@pytest.fixture(scope="module")
def reference():
    sc = _scene(3)
    return sc, {p: oracle_render(p, sc, _clear())[:2] for p in ("PixelPipe_gouraud", "PixelPipe_trihash_srcover")}


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_trihash_srcover"])
def test_more_pairs_than_records(cuda, reference, pipe):
    sc, refs = reference
    n = sc["indices"].shape[0]
    cr = pkg().CudaRaster()
    cr.init()
    for k in range(3):   # without room for all records, then with it
        c, d, cnt, _ = gpu_render(pipe, sc, _clear(), cr=cr, capacity=(2 * n, 10**8, 12 * 10**6))
        assert cnt["reruns"] == (1 if k == 0 else 0) and cnt["tile_entries"] > RECORDS + 10**6
        assert_same(c, d, *refs[pipe], f"{pipe} draw {k}")
    # The estimates' way: the first attempt overflows the tile list.
    c, d, cnt, _ = gpu_render(pipe, sc, _clear())
    assert cnt["reruns"] >= 1
    assert_same(c, d, *refs[pipe], f"{pipe} rerun")


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_trihash_srcover"])
def test_queued_draws(cuda, reference, pipe):
    sc, refs = reference
    p = pkg()
    cr = p.CudaRaster()
    cr.init()
    cr.setCapacity(10**5, 10**8, 12 * 10**6)
    s = [p.CudaSurface((SIZE, SIZE), f, 1) for f in (p.CudaSurface.FORMAT_RGBA8, p.CudaSurface.FORMAT_DEPTH32)]
    cr.setSurfaces(*s)
    cr.setPixelPipe(None, pipe)
    v, i = torch.from_numpy(sc["vertices"]).cuda(), torch.from_numpy(sc["indices"]).cuda()
    cr.setVertexBuffer(v, 0)
    cr.setIndexBuffer(i, 0, i.shape[0])
    for k in range(3):
        cr._check(cr._lib.cr_deferred_clear_raw(cr._ctx, *_clear()))
        cr.drawTrianglesAsync()
        if k == 1:   # two queued together
            continue
        torch.cuda.synchronize()
        assert cr.getCounters()["overflow"] == 0
        assert_same(*(t.download().numpy().astype(np.uint32) for t in s), *refs[pipe], f"{pipe} queued draw {k}")


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_trihash_srcover"])
def test_captured_batch_and_draws_beside_it(cuda, reference, pipe):
    sc, refs = reference
    p = pkg()
    cr = p.CudaRaster()
    cr.init()
    cr.setCapacity(10**5, 10**8, 12 * 10**6)
    s = [p.CudaSurface((SIZE, SIZE), f, 1) for f in (p.CudaSurface.FORMAT_RGBA8, p.CudaSurface.FORMAT_DEPTH32)]
    v, i = torch.from_numpy(sc["vertices"]).cuda(), torch.from_numpy(sc["indices"]).cuda()
    graph = cr.createBatchGraph([{"pipe": pipe, "color": s[0], "depth": s[1], "vertices": v, "indices": i,
                                  "numTris": i.shape[0], "clear": (0.1, 0.2, 0.3, 1.0, 1.0)}])
    for k in range(3):
        graph.launch()
        assert graph.counters()["overflow"] == 0
        assert_same(*(t.download().numpy().astype(np.uint32) for t in s), *refs[pipe], f"{pipe} replay {k}")
        # A draw beside the graph lacks records too, and must leave the graph's in place.
        c, d, cnt, _ = gpu_render(pipe, sc, _clear(), cr=cr)
        assert cnt["reruns"] == 0
        assert_same(c, d, *refs[pipe], f"{pipe} draw beside the graph {k}")
    graph.destroy()
    for _ in range(2):
        c, d, _, _ = gpu_render(pipe, sc, _clear(), cr=cr)
        assert_same(c, d, *refs[pipe], f"{pipe} after the graph")
