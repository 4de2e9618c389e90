"""8x MSAA around the triangle count up to which a visibility key has room for the
winner's coverage mask (2^21 - 1): beyond it the resolve forms edges and masks
anew. Against the oracle, exact."""
import numpy as np
import pytest

from conftest import pkg_mod
from helpers import assert_same, gpu_render, oracle_render
from test_gpu_tile_lists import _clear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2**21 - 1, 2**21])
def test_keys_with_and_without_masks(cuda, n):
    sc = dict(pkg_mod("scenes").soup(60000, 200, 150, seed=5, median_px=6.0))
    # The same triangles over and over at the end of a list of ones without area: late entries, and ties.
    idx = np.zeros((n, 3), np.int32)
    idx[-240000:] = np.tile(sc["indices"], (4, 1))
    sc["indices"] = idx
    rc, rd, st = oracle_render("PixelPipe_gouraud_msaa8", sc, _clear())
    c, d, cnt, _ = gpu_render("PixelPipe_gouraud_msaa8", sc, _clear())
    assert cnt["overflow"] == 0 and st["zmin_violations"] == 0 and cnt["num_tris"] == n
    assert_same(c, d, rc, rd, f"8x MSAA, {n} triangles")
    assert np.unique(rc).size > 1000
