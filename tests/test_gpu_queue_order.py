"""The tile lists of pipes that depend on their order, read back as the draw left
them: every list in submission order and equal to the oracle's queue model, over
list lengths from one entry to thousands; and the device's entry count of every
bin against the model."""
import numpy as np
import pytest

from conftest import pkg_mod
from helpers import PIPES, PIPE_SAMPLES, gpu_render, pkg, vertices_for
from oracle import oracle as orc
from test_gpu_queues import SCENES, _check_level, _gpu_queues
from test_gpu_tile_lists import _clear, _triangles

pytestmark = pytest.mark.gpu


def _crowded():
    """Lists of 3 to 6,000 entries (registers, shared memory, radix) on a small viewport."""
    rng = np.random.default_rng(7)
    parts = [rng.uniform(0, 90, (2000, 1, 2)) + rng.uniform(0, 9, (2000, 3, 2))]
    for n, x, y in ((300, 8, 8), (1500, 32, 16), (6000, 64, 40)):
        parts.append(np.array([[x + 0.5, y + 0.5], [x + 7.4, y + 0.5], [x + 0.5, y + 7.4]]) + rng.uniform(-0.3, 0.3, (n, 3, 2)))
    return _triangles(rng.permutation(np.concatenate(parts)), 101, 67, 8)


@pytest.mark.parametrize("pipe", ["PixelPipe_gouraud_srcover", "PixelPipe_gouraud_nodepth", "PixelPipe_deriv_quads",
                                  "PixelPipe_gouraud_srcover_msaa4", "PixelPipe_gouraud"])
@pytest.mark.parametrize("scene", [*SCENES, "crowded"])
def test_lists_and_bin_counts(cuda, pipe, scene):
    lib = pkg_mod("_lib").load()
    sc = _crowded() if scene == "crowded" else SCENES[scene]()
    cr = pkg().CudaRaster()
    cr.init()
    gpu_render(pipe, sc, _clear(), cr=cr)
    (_, bin_count, _), tiles = _gpu_queues(cr, lib)
    flags, blend, shader, stride = PIPES[pipe]
    op = orc.make_pipe(sc["width"], sc["height"], PIPE_SAMPLES.get(pipe, 1), flags, blend, shader, stride)
    q = {k: orc.queue_lists(op, vertices_for(pipe, sc["vertices"]), sc["indices"], 4, k) for k in orc.QUEUE_KINDS}
    _check_level("tile", tiles, q["tile_exact"], q["tile_rule"], f"{pipe} {scene}")
    assert np.array_equal(bin_count, np.diff(q["bin_rule"][0]))
