// Entry of the tile rings of the grouped GEMMs: the publisher of a CTA's tile schedule hands each tile to the other warps
// through a slot of shared memory that is written again 32 tiles later.
//
// An entry is two 64-bit words and each of them carries the tile's sequence number.  PTX gives single-copy atomicity
// to scalar accesses of up to 64 bits; a vector access counts as scalar ones in no particular order.  So a reader that finds its
// number in BOTH words has the whole tile, whichever word arrived first, with one vector load and no fence (a
// number in one word of four, as it was, promises nothing about the other three).
// Plain C++ as well: the CPU tests compile it.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define B200MOE_HD __host__ __device__ __forceinline__
#else
#define B200MOE_HD inline
#endif

namespace b200moe {

constexpr int kTileRing = 32;

struct TileEntry {
    uint64_t a;  // sequence number (32 bits) | first row << 32
    uint64_t b;  // low 16 bits of the sequence number | rows << 16 (9 bits) | expert << 25 (11 bits) | tile column << 36
};

// rows 1 .. 256, g < 1024 experts, column of 256 weight columns < 2^23; rows 0: the schedule has ended.
B200MOE_HD TileEntry tile_entry(uint32_t seq, uint32_t row0, uint32_t rows, uint32_t g, uint32_t column) {
    TileEntry e;
    e.a = seq | ((uint64_t)row0 << 32);
    e.b = (uint64_t)((seq & 0xFFFFu) | (rows << 16)) | ((uint64_t)g << 25) | ((uint64_t)column << 36);
    return e;
}
// Whether both words are those of the seq-th tile.  A slot's earlier numbers differ by multiples of 32 and its reader
// is never a whole ring behind, so 16 bits tell them apart as well as 32 do.
B200MOE_HD bool tile_entry_is(const TileEntry& e, uint32_t seq) {
    return (uint32_t)e.a == seq && (((uint32_t)e.b ^ seq) & 0xFFFFu) == 0;
}
B200MOE_HD int tile_entry_row0(const TileEntry& e) { return (int)(e.a >> 32); }
B200MOE_HD int tile_entry_rows(const TileEntry& e) { return (int)(((uint32_t)e.b >> 16) & 0x1FFu); }
B200MOE_HD int tile_entry_expert(const TileEntry& e) { return (int)((uint32_t)(e.b >> 25) & 0x7FFu); }
B200MOE_HD int tile_entry_column(const TileEntry& e) { return (int)(e.b >> 36); }

}  // namespace b200moe

#ifdef __CUDACC__
#include "ptx.cuh"
namespace b200moe {
__device__ __forceinline__ TileEntry ring_load(const TileEntry* e) {
    TileEntry v;
    asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "r"(ptx::smem_u32(e)));
    return v;
}
__device__ __forceinline__ void ring_store(TileEntry* e, const TileEntry& v) {
    asm volatile("st.volatile.shared.v2.u64 [%0], {%1, %2};" ::"r"(ptx::smem_u32(e)), "l"(v.a), "l"(v.b) : "memory");
}
}  // namespace b200moe
#endif
