"""The tile hand-off of the grouped GEMMs (csrc/tile_ring.h), compiled for the host: a reader of a ring slot sees each of an
entry's two words at any time before or after it was written, and must not take a mixture for a tile."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ascend_kernel_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "tile_ring.h"
using namespace b200moe;

struct Tile { uint32_t row0, rows, g, column; };

int main() {
    // corners of every field, the end of the schedule among them
    const Tile tiles[] = {{0, 1, 0, 0}, {0x7FFFFFEF, 256, 1023, 0x7FFFFF}, {128, 128, 1, 1}, {5, 0, 0, 0}, {255, 160, 512, 27}, {0, 32, 1023, 0}};
    const uint32_t seqs[] = {1, 2, 31, 32, 33, 64, 4097, 65535, 65536, 65537, 65568, 0x7FFFFFFF, 0xFFFFFFE0u};
    for (uint32_t seq : seqs)
        for (const Tile& t : tiles) {
            const TileEntry now = tile_entry(seq, t.row0, t.rows, t.g, t.column);
            if (!tile_entry_is(now, seq)) return std::printf("entry %u does not carry its number\n", seq), 1;
            if (tile_entry_row0(now) != (int)t.row0 || tile_entry_rows(now) != (int)t.rows ||
                tile_entry_expert(now) != (int)t.g || tile_entry_column(now) != (int)t.column)
                return std::printf("entry %u is not the tile that went in\n", seq), 1;
            // what the slot held before: nothing, or the tile of one to four rounds earlier
            for (uint32_t back = 0; back <= 4; ++back) {
                if (back && seq <= back * kTileRing) continue;
                for (const Tile& o : tiles) {
                    const TileEntry was = back ? tile_entry(seq - back * kTileRing, o.row0, o.rows, o.g, o.column) : tile_entry(0, 0, 0, 0, 0);
                    TileEntry torn[3] = {{now.a, was.b}, {was.a, now.b}, was};
                    // (the empty slot's 16 bits are those of tile 65536, which comes when it has been written 2047 times)
                    for (const TileEntry& e : torn)
                        if (!(back == 0 && seq % 65536 == 0) && tile_entry_is(e, seq))
                            return std::printf("a mixture passes for tile %u\n", seq), 1;
                }
            }
        }
    return 0;
}
"""


def test_a_half_written_entry_is_never_a_tile(tmp_path):
    src, exe = tmp_path / "ring.cpp", tmp_path / "ring"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("name", ["grouped_gemm.cu", "grouped_gemm_packed.cu"])
def test_both_kernels_hand_tiles_over_through_it(name):
    """No vector access of 32-bit words with a flag among them: PTX promises nothing about the order of its elements."""
    text = open(os.path.join(CSRC, name)).read()
    assert "ring_store(&sb->tile_ring[" in text and "ring_load(e)" in text
    assert not re.search(r"volatile\.shared\.v4", text)
