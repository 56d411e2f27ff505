"""Chunk positions and midpoints at the largest CSRs (2^31 - 1 entries), compiled for the
host and compared with Python's integers."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "graphhet_b200", "csrc")
SOURCE = """
#include "row_math.cuh"
extern "C" int32_t count(int32_t len, int32_t size) { return ghb::chunk_count(len, size); }
extern "C" int32_t end(int32_t at, int32_t size, int32_t e) { return ghb::chunk_end(at, size, e); }
extern "C" int32_t middle(int32_t lo, int32_t hi) { return ghb::row_middle(lo, hi); }
"""
TOP = 2**31 - 1


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("row_math")
    (d / "f.cpp").write_text(SOURCE)
    so = str(d / "f.so")
    subprocess.run(["g++", "-O2", "-fwrapv", "-shared", "-fPIC", "-I", CSRC, str(d / "f.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("size", [32, 128])
def test_chunks_up_to_the_last_entry(host, size):
    for length in [0, 1, size - 1, size, size + 1, 4 * size + 3, TOP - size, TOP - 1, TOP]:
        assert host.count(length, size) == -(-length // size)
    for end in [1, size, size + 5, 2**30, TOP - size, TOP - 1, TOP]:
        for at in [max(0, end - k) for k in (1, 2, size - 1, size, size + 1, 3 * size)]:
            assert host.end(at, size, end) == min(end, at + size)


def test_midpoints_past_2_30(host):
    for hi in [0, 1, 7, 2**30, 2**30 + 1, TOP - 1, TOP]:
        for lo in [0, hi // 2, max(0, hi - 9), max(0, hi - 1), hi]:
            assert host.middle(lo, hi) == (lo + hi) // 2
