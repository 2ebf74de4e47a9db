"""How launches are cut into CTAs (garnet_b200/csrc/launch_plan.h), compiled for the host."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "garnet_b200", "csrc")
SHIM = """
#include "launch_plan.h"
using namespace gb200;
extern "C" void tile_plan(int panels, int chunks, int m, int* out)
{
    const TcPlan t = tc_plan(panels * 8, chunks, m);
    out[0] = t.row_tiles, out[1] = t.tile_rows, out[2] = t.kslices;
    for (int s = 0; s <= t.kslices; ++s) out[3 + s] = tc_first_chunk(chunks, t.kslices, s);
}
extern "C" int prefill_tiles(int batch, int kv_heads, int tokens, int tile_tokens) { return oss_prefill_tiles(batch, kv_heads, tokens, tile_tokens); }
"""
SMS = 148


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    path = tmp_path_factory.mktemp("plan")
    (path / "shim.cpp").write_text(SHIM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(path / "shim.cpp"), "-o", str(path / "shim.so")])
    return ctypes.CDLL(str(path / "shim.so"))


@pytest.mark.parametrize("m", [17, 64, 77, 192, 193, 400, 1000])
def test_tile_kernel_keeps_its_k_slices_whatever_the_chunk_count(plans, m):
    """Every K that has two chunks is cut while the tiles leave half of the SMs idle; the slices cover K without a gap, none
    is empty and the longest has at most one chunk more than the shortest."""
    out = (ctypes.c_int * 16)()
    for panels in (1, 2, 4, 8, 16, 32, 48, 74, 75, 96, 148, 1187):
        for chunks in range(1, 90):
            plans.tile_plan(panels, chunks, m, out)
            row_tiles, tile_rows, slices = out[:3]
            assert row_tiles * tile_rows >= m > (row_tiles - 1) * tile_rows and tile_rows % 16 == 0 and tile_rows <= 192
            tiles = panels * row_tiles
            assert slices == 1 or tiles * slices <= SMS
            assert slices > 1 or chunks == 1 or 2 * tiles > SMS, (panels, chunks)
            if tile_rows > 96:     # a CTA has an SM for itself: that many clusters of the size run at once on a B200
                assert slices == 1 or tiles <= {2: 74, 4: 33, 8: 15}[slices]
            first = out[3:4 + slices]
            sizes = [b - a for a, b in zip(first, first[1:])]
            assert first[0] == 0 and first[-1] == chunks and min(sizes) >= 1 and max(sizes) - min(sizes) <= 1


def test_prefill_takes_a_second_query_tile_only_where_there_is_one(plans):
    """A CTA takes two tiles when they hold rows and the CTAs still fill the GPU."""
    plans.prefill_tiles.restype = ctypes.c_int
    for batch in (1, 2, 3, 7, 20, 64):
        for kv_heads, tile_tokens in ((8, 16), (1, 16), (8, 128), (2, 42), (16, 1)):
            for tokens in list(range(1, 70)) + [128, 129, 700, 2048, 65000]:
                tiles = plans.prefill_tiles(batch, kv_heads, tokens, tile_tokens)
                blocks = -(-tokens // (2 * tile_tokens))
                assert tiles == (2 if tokens > tile_tokens and batch * kv_heads * blocks >= SMS else 1)
