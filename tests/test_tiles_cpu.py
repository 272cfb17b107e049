"""Roots per tile of a search launch (everest_b200/csrc/evx_tiles.h, compiled
for the host): the tiles of a launch are numbered in an int, with room for the
claims past the end, whatever the batch holds; launches that fit keep the
finer tiles."""
import ctypes
import subprocess

import pytest

from everest_b200 import autotune, build

INT_MAX = 2**31 - 1
MAX_EDGES = 2**30 - 2
WRAP = """
#include "evx_tiles.h"
extern "C" int roots_of(int k, long long roots, long long queries, long long warps, int most) {
  return evx::tile_roots_for(k, roots, queries, warps, most);
}
extern "C" long long tiles_of(long long roots, int tile) { return evx::tiles_of(roots, tile); }
"""


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiles")
    (d / "t.cc").write_text(WRAP)
    subprocess.run([build._cxx(), "-shared", "-fPIC", "-std=c++17", "-I", build.CSRC, "-o", str(d / "t.so"), str(d / "t.cc")],
                   check=True)
    lib = ctypes.CDLL(str(d / "t.so"))
    ll, i = ctypes.c_longlong, ctypes.c_int
    lib.roots_of.argtypes, lib.roots_of.restype = [i, ll, ll, ll, i], i
    lib.tiles_of.argtypes, lib.tiles_of.restype = [ll, i], ll
    return lib


@pytest.mark.parametrize("queries,roots", [
    (1, 1), (1, MAX_EDGES), (64, 250_000), (1908, 36_000_000 - 3), (1910, 36_000_000 - 3), (15_272, 36_000_000 - 3),
    (138, 500_000_000), (1100, 500_000_000), (1 << 20, 1), (1 << 20, 3000), (1 << 20, MAX_EDGES)])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 8])
@pytest.mark.parametrize("bps", [1, 10, 1000])
def test_tile_numbers_fit(tiles, k, queries, roots, bps):
    warps = bps * 148 * 4
    for most in (32, 256, 1 << 20):
        tile = tiles.roots_of(k, queries * roots, queries, warps, most)
        assert 1 <= tile <= 1 << 29
        assert queries * tiles.tiles_of(roots, tile) + 2 * warps <= INT_MAX
        cap = min(most, 32 if k == 4 else 64)
        if queries * tiles.tiles_of(roots, cap) < INT_MAX // 2:
            assert tile <= cap


def test_no_room(tiles):
    assert tiles.roots_of(4, 1000, 1, 1 << 30, 64) == 0


def test_tuned_batch_tiles_differ(tiles):
    # what the tuner times are different tilings of a range that fills the GPU
    got = [tiles.roots_of(3, 1 << 30, 64, 5920, most) for most in autotune.BATCH_TILES]
    assert got == list(autotune.BATCH_TILES)
