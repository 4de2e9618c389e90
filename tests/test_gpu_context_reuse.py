"""One context for draws of changing sizes: its list arrays share two
allocations, whose pieces move from draw to draw, one of them zero between
draws. Every draw must equal a fresh context's, also after an overflow and
beside a captured graph that holds the pieces of an earlier draw."""
import numpy as np
import pytest
import torch

from conftest import pkg_mod
from helpers import assert_same, gpu_render, oracle_render, pkg
from test_gpu_batch import _batch_scenes, _clear, _instances

pytestmark = pytest.mark.gpu


def _words(s):
    return s.download().numpy().astype(np.uint32)


def _scenes():
    soup = pkg_mod("scenes").soup
    return [("PixelPipe_gouraud", soup(20000, 64, 64, seed=1, median_px=4.0)),
            ("PixelPipe_gouraud_srcover", soup(300, 1500, 900, seed=2, median_px=200.0, alpha_range=(0.2, 1.0))),
            ("PixelPipe_gouraud_msaa4", soup(5, 33, 700, seed=3, median_px=30.0)),
            ("PixelPipe_gouraud", soup(40000, 1400, 1000, seed=4, median_px=6.0)),
            ("PixelPipe_gouraud_nodepth", soup(9000, 40, 24, seed=5, median_px=12.0)),
            ("PixelPipe_gouraud", soup(1, 8, 8, seed=6))]


def test_draws_of_changing_sizes(cuda):
    cr = pkg().CudaRaster()
    cr.init()
    refs = [oracle_render(pipe, sc, _clear())[:2] for pipe, sc in _scenes()]
    order = [0, 1, 2, 3, 4, 5, 3, 0, 4, 1, 5, 2]
    for k in order:
        pipe, sc = _scenes()[k]
        c, d, cnt, _ = gpu_render(pipe, sc, _clear(), cr=cr)
        assert cnt["overflow"] == 0
        assert_same(c, d, *refs[k], f"scene {k} ({pipe}) on a used context")


def test_an_overflow_leaves_the_arrays_zero(cuda):
    """A queued draw that overflows its subtriangles, then one that overflows its tile list, each before a good one."""
    sc = pkg_mod("scenes").soup(6000, 256, 200, seed=9, median_px=100.0)
    v = sc["vertices"].copy()
    v[::7, 2] = -1.5 * v[::7, 3]
    sc["vertices"] = v
    ref = oracle_render("PixelPipe_gouraud", sc, _clear())[:2]
    for capacity in ((6000, 10**7, 10**7), (10**5, 10**7, 1000)):
        cr = pkg().CudaRaster()
        cr.init()
        cr.setCapacity(*capacity)
        p = pkg()
        s = [p.CudaSurface((256, 200), f, 1) for f in (p.CudaSurface.FORMAT_RGBA8, p.CudaSurface.FORMAT_DEPTH32)]
        cr.setSurfaces(*s)
        cr.setPixelPipe(None, "PixelPipe_gouraud")
        vt, it = torch.from_numpy(v).cuda(), torch.from_numpy(sc["indices"]).cuda()
        cr.setVertexBuffer(vt, 0)
        cr.setIndexBuffer(it, 0, it.shape[0])
        cr._check(cr._lib.cr_deferred_clear_raw(cr._ctx, *_clear()))
        cr.drawTrianglesAsync()
        torch.cuda.synchronize()
        assert cr.getCounters()["overflow"] != 0
        c, d, cnt, _ = gpu_render("PixelPipe_gouraud", sc, _clear(), cr=cr)
        assert cnt["overflow"] == 0 and cnt["reruns"] >= 1
        assert_same(c, d, *ref, f"after an overflow of {capacity}")


def test_draws_beside_a_captured_graph(cuda):
    """Draws no array of which needs more than the batch's, nor than an earlier draw's, leave the graph's memory."""
    soup = pkg_mod("scenes").soup
    many, wide = soup(60000, 64, 64, seed=11, median_px=3.0), soup(100, 1000, 800, seed=12, median_px=60.0)
    both = dict(soup(60000, 1000, 800, seed=13, median_px=3.0))
    cr = pkg().CudaRaster()
    cr.init()
    for sc in (many, wide):
        gpu_render("PixelPipe_gouraud", sc, _clear(), cr=cr)
    items = _batch_scenes()
    insts, keep = _instances(items, (0.1, 0.2, 0.3, 1.0, 1.0))
    refs = [gpu_render(pipe, sc, _clear())[:2] for pipe, sc in items]
    cr.drawBatch(insts)
    graph = cr.createBatchGraph(insts)
    other = oracle_render("PixelPipe_gouraud", both, _clear())[:2]
    for _ in range(2):
        c, d, _, _ = gpu_render("PixelPipe_gouraud", both, _clear(), cr=cr)
        assert_same(c, d, *other, "draw beside the graph")
        graph.launch()
        assert graph.counters()["overflow"] == 0
        for (rc, rd), (cs, ds, _, _) in zip(refs, keep):
            assert_same(_words(cs), _words(ds), rc, rd, "graph replay beside draws")
    graph.destroy()
