"""The resolve at the widths where its 128-pixel lines and 4-pixel loads end,
with output rows at every word offset, and from a surface that starts off a
16-byte boundary (the scalar kernel). Exact against the rule."""
import ctypes as C

import numpy as np
import pytest

from conftest import pkg_mod
from test_resolve import resolve_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset_words", [0, 1])
@pytest.mark.parametrize("samples", [1, 2, 4, 8])
@pytest.mark.parametrize("width,height", [(1, 1), (4, 3), (5, 8), (127, 9), (128, 2), (129, 7), (255, 5), (4095, 3)])
def test_resolve_edges(cuda, width, height, samples, offset_words):
    torch = cuda
    lib = pkg_mod("_lib").load()
    rows, words = (height + 7) & ~7, ((width + 7) & ~7) * samples
    g = torch.Generator(device="cuda").manual_seed(width * 31 + height)
    buf = torch.randint(-2**31, 2**31 - 1, (rows * words + 4,), generator=g, device="cuda", dtype=torch.int32)
    surf = buf[offset_words:offset_words + rows * words]
    pitch = width + 3          # output rows at all word offsets
    out = torch.full((height, pitch), 7, dtype=torch.int32, device="cuda")
    assert lib.cr_resolve_color(surf.data_ptr(), width, height, samples, out.data_ptr(), pitch * 4,
                                C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    want = resolve_reference(surf.cpu().numpy().view(np.uint32).reshape(rows, words), width, height, samples)
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[:, :width].copy().view(np.uint8).reshape(height, width, 4), want)
    assert (got[:, width:] == 7).all()
