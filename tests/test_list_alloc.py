"""The arithmetic that allocates the tile lists (include/cudaraster/detail/
list_alloc.h), compiled with the host compiler: totals beyond 2^31 entries are
found not to fit instead of wrapping, and no index outside the list memory is
accepted."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
I32_MAX = 2**31 - 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("list_alloc") / "list_alloc.so"
    cmd = ["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-shared", "-fPIC", f"-I{ROOT / 'include'}",
           str(ROOT / "tests" / "cpp" / "list_alloc.cpp"), "-o", str(so)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    lib = C.CDLL(str(so))
    lib.group_entries.argtypes, lib.group_entries.restype = [C.c_void_p], C.c_uint64
    lib.group_fits.argtypes, lib.group_fits.restype = [C.c_void_p, C.c_uint64, C.c_int64], C.c_int32
    lib.reported.argtypes, lib.reported.restype = [C.c_uint64], C.c_int32
    lib.holds.argtypes, lib.holds.restype = [C.c_int32, C.c_int64], C.c_int32
    return lib


# Counts per tile whose 1,024-fold sum wraps a 32-bit total to a negative, a zero and a small positive value.
@pytest.mark.parametrize("count", [1, 100, 2**21 - 1, 2**21, 3145728, 2**22 - 1, 2**22, 2**22 + 7, 2**23 + 1, 2**29 - 1])
@pytest.mark.parametrize("before", [0, 1, I32_MAX, 2**32 - 5, 2**40])
def test_groups_beyond_the_capacity_do_not_fit(lib, count, before):
    counts = np.full(1024, count, np.int32)
    total = 1024 * count
    assert lib.group_entries(counts.ctypes.data) == total
    for capacity in (1, 102400, total - 1, total, total + before - 1, total + before, I32_MAX, 2**31, 2**40):
        fits = lib.group_fits(counts.ctypes.data, before, capacity)
        assert fits == (before + total <= min(capacity, I32_MAX)), (count, before, capacity)


def test_uneven_counts(lib):
    rng = np.random.default_rng(1)
    for _ in range(200):
        counts = (rng.uniform(0, 1, 1024) ** 8 * 2**29).astype(np.int32)
        total = int(counts.astype(np.int64).sum())
        assert lib.group_entries(counts.ctypes.data) == total
        assert lib.reported(total) == min(total, I32_MAX)


@pytest.mark.parametrize("index", [-2**31, -2**30, -1, 0, 1, 999, 1000, 2**30, I32_MAX])
@pytest.mark.parametrize("capacity", [1, 1000, I32_MAX, 2**31, 2**32, 2**40])
def test_list_indices(lib, index, capacity):
    assert lib.holds(index, capacity) == (0 <= index < capacity)
