"""The memory that getProfilingInfo reports is what the context has allocated, and
the fly-through's list memory is read from it."""
import re

import pytest
import torch

from conftest import pkg_mod
from helpers import gpu_render, pkg
from test_gpu_tile_lists import _clear

pytestmark = pytest.mark.gpu


def _mb(text, name):
    return float(re.search(name + r"\s+([0-9.]+) MB", text).group(1))


def _held_outside_torch():
    """Device memory in use except torch's own (the scene's buffers, which the context refers to)."""
    free, total = torch.cuda.mem_get_info()
    return total - free - torch.cuda.memory_reserved()


def test_reported_memory_is_allocated_memory(cuda):
    sc = pkg_mod("scenes").soup(200000, 640, 480, seed=1, median_px=4.0)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cr = pkg().CudaRaster()
    cr.init()
    gpu_render("PixelPipe_gouraud", sc, _clear(), cr=cr, num_tris=1)
    torch.cuda.empty_cache()
    held0, first = _held_outside_torch(), cr.getProfilingInfo()
    _, _, cnt, _ = gpu_render("PixelPipe_gouraud", sc, _clear(), cr=cr)
    torch.cuda.empty_cache()
    text = cr.getProfilingInfo()
    grown = (_held_outside_torch() - held0) / 2**20
    # cudaMalloc takes whole 2 MB blocks: seven growing buffers.
    reported = _mb(text, "Scratch") - _mb(first, "Scratch")
    assert reported > 20.0
    assert abs(grown - reported) <= 2 * 7 + 1, (grown, reported)
    n = 200000
    lists = 16 * n + 8 * n + 4 * cnt["max_tile_entries"] + 8 * cnt["max_tile_entries"]
    assert lists / 2**20 <= _mb(text, "List memory") <= _mb(text, "Scratch") - 80 * n / 2**20
    assert not re.search(r"Bin entries.*MB", text)


def test_flythrough_list_memory(cuda):
    wl = pkg_mod("workloads")
    cr = pkg().CudaRaster()
    cr.init()
    gpu_render("PixelPipe_gouraud", pkg_mod("scenes").soup(1000, 64, 64, seed=2), _clear(), cr=cr)
    assert wl.list_memory_mb(cr) == _mb(cr.getProfilingInfo(), "List memory") > 0.0
