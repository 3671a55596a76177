"""Every layout the binned sweep can choose stays inside its buffer: bins and
spill area within the rows of the buffer, no more spilled rows than spill tags,
counters within their set.  Walked over buffer sizes, row counts, growth and
the rows a block holds at each key width, against the rule itself compiled for
the host (tests/bin_layout_host.cpp)."""

from __future__ import annotations

import ctypes
import itertools
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    so = tmp_path_factory.mktemp("layout") / "liblayout.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(HERE / "bin_layout_host.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(so))
    F, U = ctypes.c_float, ctypes.c_uint32
    lib.bl_layout.argtypes = [F, F, F, U, U, U, ctypes.c_uint64, ctypes.c_void_p]

    def run(n, grow, fill, rows, room):
        out = (ctypes.c_uint64 * 6)()
        lib.bl_layout(n, grow, fill, 296, 8, rows, room, out)
        return list(out)

    return run


def test_no_layout_leaves_its_buffer(layout):
    rooms = [1 << 20, (1 << 20) + 12345, 1 << 21, 3 << 20, 1 << 22, 1 << 24, (1 << 26) - 1, 1 << 30]
    ns = [0.0, 1.0, 3e3, 2.9e4, 1e5, 9.7e5, 1e6, 3.3e7, 1e8, 2.0**31]
    seen = set()
    for rows, room, n, grow, fill in itertools.product([3328, 2560, 2048, 1152], rooms, ns,
                                                       [1.0, 1.3, 2.0, 7.0, 25.0, 512.5], [0.3, 0.7, 0.85, 1.0]):
        bins, stride, cap, spills, tags, count_words = layout(n, grow, fill, rows, room)
        assert 1 <= bins and 1 <= cap
        assert bins * stride <= count_words
        assert bins * cap + spills <= room
        assert spills <= tags, f"{spills} rows may spill, {tags} tags: rows {rows} room {room} n {n} grow {grow}"
        assert spills >= room // 16  # the share set aside is always usable
        seen.add(bins)
    assert min(seen) <= 296 and max(seen) == 1 << 18


def test_a_small_buffer_with_very_many_bins(layout):
    # 2^20 rows in 70,218 bins: the bins leave 135,742 rows, 131,072 have tags
    n = 1.0e6
    bins, _, cap, spills, tags, _ = layout(n, 24.2677, 0.3, 1152, 1 << 20)
    assert abs(bins - 70218) < 100 and (1 << 20) - bins * cap > tags
    assert spills == tags == 1 << 17
