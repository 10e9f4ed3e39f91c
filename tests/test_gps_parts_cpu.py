"""How the points of a binned point-splatting Gaussian are dealt out (csrc/sgs_gps_parts.h), compiled for the host.

A caller may set any point cap below 2^32, so that counts reach 2^32 - 1: their chunks and items must cover every
point once, without a wrap of the 32-bit arithmetic, and in a bounded number of items.
"""
import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "stochastic-gaussian-splatting_b200" / "csrc"

SOURCE = """
#include "sgs_gps_parts.h"
extern "C" uint32_t chunks(uint32_t count) { return sgs::gps_chunks(count); }
extern "C" uint32_t parts(uint32_t count) { return sgs::gps_parts(count).parts; }
extern "C" uint32_t points(uint32_t count) { return sgs::gps_parts(count).points; }
extern "C" uint32_t item_first(uint32_t count, uint32_t part) { return sgs::gps_item_points(count, part).first; }
extern "C" uint32_t item_n(uint32_t count, uint32_t part) { return sgs::gps_item_points(count, part).n; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    folder = tmp_path_factory.mktemp("gps_parts")
    (folder / "parts.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC), str(folder / "parts.cpp"), "-o",
                    str(folder / "parts.so")], check=True)
    lib = ctypes.CDLL(str(folder / "parts.so"))
    for f in (lib.chunks, lib.parts, lib.points, lib.item_first, lib.item_n):
        f.restype, f.argtypes = ctypes.c_uint32, [ctypes.c_uint32] * (2 if "item" in f.__name__ else 1)
    return lib


EDGES = [513, 2047, 2048, 2049, 1024 * 2048, 1024 * 2048 + 1, 1023 << 22, (1023 << 22) + 1, (1 << 32) - 4096,
         (1 << 32) - 257, (1 << 32) - 256, (1 << 32) - 255, (1 << 32) - 129]
WRAPPING = [(1 << 32) - 2047, (1 << 32) - 128, (1 << 32) - 1]


@pytest.mark.parametrize("count", EDGES + WRAPPING)
def test_chunks_cover_every_point(lib, count):
    assert lib.chunks(count) == -(-count // 256)


@pytest.mark.parametrize("count", EDGES + WRAPPING)
def test_items_cover_every_point_once(lib, count):
    assert lib.points(count) > 0
    parts = lib.parts(count)
    assert 1 <= parts <= 1024
    at = 0
    for part in range(parts):
        assert lib.item_first(count, part) == at
        n = lib.item_n(count, part)
        assert 1 <= n <= 1 << 22  # the consumer's strided loop over n points cannot wrap
        at += n
    assert at == count


def test_an_unused_entry_has_none(lib):
    assert lib.chunks(0) == 0 and lib.parts(0) == 0
