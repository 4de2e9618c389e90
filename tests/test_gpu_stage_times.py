"""The stage times of getStats: with stage timing on they are positive, in
seconds and together the draw's; off they are zero; a draw without triangles
has none before its lists."""
import numpy as np
import pytest
import torch

from conftest import pkg_mod
from helpers import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris", [0, 1, 5000, 300000])
@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_gouraud_srcover"])
def test_stage_times_add_up(cuda, pipe, tris):
    p = pkg()
    sc = pkg_mod("scenes").soup(max(tris, 1), 640, 480, seed=3)
    size = (640, 480)
    cr = p.CudaRaster()
    cr.init()
    cr.setSurfaces(p.CudaSurface(size, p.CudaSurface.FORMAT_RGBA8), p.CudaSurface(size, p.CudaSurface.FORMAT_DEPTH32))
    cr.setPixelPipe(None, pipe)
    cr.setVertexBuffer(torch.from_numpy(np.ascontiguousarray(sc["vertices"][:, :8])).cuda(), 0)
    cr.setIndexBuffer(torch.from_numpy(sc["indices"]).cuda(), 0, tris)
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for queued in (False, True):
        for _ in range(3):
            cr.deferredClear((0.1, 0.2, 0.3, 1.0), 1.0)
            a.record()
            cr.drawTrianglesAsync() if queued else cr.drawTriangles()
            b.record()
            s = cr.getStats()
        torch.cuda.synchronize()
        t = [s.setupTime, s.binTime, s.coarseTime, s.fineTime]
        assert all(x >= 0.0 for x in t) and t[3] > 0.0
        if tris:
            assert min(t) > 0.0
        # The events around the call hold the draw's block and the event records besides.
        assert sum(t) <= a.elapsed_time(b) * 1e-3 + 2e-6
    cr.setStageTiming(False)
    cr.drawTriangles()
    s = cr.getStats()
    assert [s.setupTime, s.binTime, s.coarseTime, s.fineTime] == [0.0] * 4


def test_batch_whose_first_pipe_has_no_triangles(cuda):
    """The first setup launch is the second pipe's: its time still counts as setup."""
    p = pkg()
    sc = pkg_mod("scenes").soup(200000, 640, 480, seed=4)
    v, i = torch.from_numpy(np.ascontiguousarray(sc["vertices"][:, :8])).cuda(), torch.from_numpy(sc["indices"]).cuda()
    insts = [{"pipe": pipe, "color": p.CudaSurface((640, 480), p.CudaSurface.FORMAT_RGBA8),
              "depth": p.CudaSurface((640, 480), p.CudaSurface.FORMAT_DEPTH32), "vertices": v, "indices": i,
              "numTris": n, "clear": (0.1, 0.2, 0.3, 1.0, 1.0)}
             for pipe, n in (("PixelPipe_gouraud", 0), ("PixelPipe_gouraud_srcover", 200000))]
    cr = p.CudaRaster()
    cr.init()
    cr.drawBatch(insts)
    s = cr.getStats()
    assert min(s.setupTime, s.binTime, s.coarseTime, s.fineTime) > 0.0
