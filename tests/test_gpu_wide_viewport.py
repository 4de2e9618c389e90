"""Viewports beyond the fast path's bound (2^15 - 1 subpixels over x and y
together): triangles of two corners take the clipper's path without a plane
cutting them, beside fast-path and cut ones. Framebuffers and the setup
stage's words against the oracle, exact."""
import ctypes as C

import numpy as np
import pytest

from conftest import pkg_mod
from helpers import PIPES, PIPE_SAMPLES, assert_same, gpu_render, oracle_render, pkg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud", "PixelPipe_gouraud_srcover", "PixelPipe_gouraud_msaa4"])
@pytest.mark.parametrize("size", [(4095, 2161), (2049, 4094), (2050, 2050)])
def test_corner_triangles_match_the_oracle(cuda, pipe, size):
    w, h = size
    sc = pkg_mod("scenes").soup(6000, w, h, seed=w + h, median_px=14.0, sigma=1.2)
    v = sc["vertices"].reshape(-1, 3, 8)
    v[::11, 0, 2] = -1.4 * v[::11, 0, 3]     # through the near plane
    v[5::17, 1, 0] *= 1.5                    # some through a side plane
    sc["vertices"] = v.reshape(-1, 8)
    p = pkg()
    clear = (p.color_to_abgr(0.1, 0.2, 0.3, 1.0), p.clear_depth_from_float(1.0))
    cr = p.CudaRaster()
    cr.init()
    c, d, cnt, _ = gpu_render(pipe, sc, clear, cr=cr)
    rc, rd, st = oracle_render(pipe, sc, clear)
    assert cnt["overflow"] == 0 and st["zmin_violations"] == 0
    assert_same(c, d, rc, rd, f"{pipe} {w}x{h}")
    # Setup words of the triangles with one subtriangle.
    flags, blend, shader, stride = PIPES[pipe]
    op = orc.make_pipe(w, h, PIPE_SAMPLES.get(pipe, 1), flags, blend, shader, stride)
    osub, ohdr, odata, _ = orc.setup(op, sc["vertices"], sc["indices"])
    n = cnt["num_subtris"]
    sub, hdr, data = np.zeros(6000, np.uint8), np.zeros((n, 4), np.uint32), np.zeros((n, 16), np.uint32)
    nt, ns = C.c_int64(), C.c_int64()
    assert pkg_mod("_lib").load().cr_read_setup_output(cr._ctx, sub.ctypes.data, hdr.ctypes.data, data.ctypes.data, n,
                                                       C.byref(nt), C.byref(ns)) == 0
    assert np.array_equal(sub, osub)
    one = np.flatnonzero(sub == 1)
    assert one.size > 1000
    assert np.array_equal(hdr[one], ohdr[one]) and np.array_equal(data[one], odata[one])
