// Antiquant grouped GEMM for prefill-sized expert batches: persistent, warp-specialised
// tcgen05 / TMEM kernel fed by TMA (sm_100a).
//
//   y[rows of expert g] = bf16( x[rows of expert g] @ dequant(W[g]) ),  fp32 accumulation in TMEM.
//
// One CTA per SM draws output tiles of up to 256 rows x 256 columns from a global ticket counter:
// two UMMA 128x256x16 instructions (rows 0-127 and 128-255 of the tile, one TMEM accumulator of
// 256 columns each) share every dequantised weight stage, so the CUDA-core dequant work per
// tensor-core flop is half that of a 128-row tile; tiles with at most 128 rows issue one.  The
// tile list is derived inside the kernel from the device-side group_list (prefix sum over the
// experts' tile counts kept in shared memory, binary search per tile), so there is no host
// synchronisation and no schedule in global memory.
//
// Warp roles (28 warps):
//   warp 0      TMA producer of x tiles (one or two boxes of 128 rows x 64 k, bf16, 128-byte
//               swizzle, K-major A) and L2 prefetch of the packed weight tiles further ahead
//   warp 2      TMEM allocation + tcgen05.mma issue (one elected lane)
//   warps 4-11  epilogue, four warps per accumulator: tcgen05.ld, scale/offset in fp32, bf16 stores
//   warps 12-27 dequant, two groups of 8 warps taking alternate k-stages: packed weights global ->
//               registers (128-bit coalesced loads, prefetched two of the group's stages ahead) ->
//               bf16 tile in the UMMA MN-major 128-byte-swizzle layout
// One ring of 3 stages (x boxes 32 KB + bf16 weights 32 KB), one full and one empty barrier per
// stage: the MMA warp pays one wait and one commit per stage.  Shared-memory bandwidth bounds this kernel (the
// tensor core alone reads 48 KB per 64-k stage), so packed weights go through registers, not
// through a shared-memory staging ring, and the bf16 tile is written without bank conflicts.
// Weights never make a round trip through global memory.  Every wait is bounded; on expiry the
// kernel records an error status, all roles wind down, copies in flight are given time to land
// and TMEM is released.
#include <cuda_fp16.h>

#include <mutex>

#include "common.cuh"
#include "gemm_args.cuh"
#include "ptx.cuh"
#include "tile_ring.h"

namespace b200moe {

constexpr int kBM = 128, kBN = 256, kBK = 64;
constexpr int kTileM = 2 * kBM;  // rows of an output tile (two MMA row halves)
constexpr int kNS = 3;  // ring stages, each an x stage (32 KB) and a bf16 weight stage (32 KB); int4: 2 stages of 32 + 2 x 32 KB
constexpr int kPrefetch = 2;  // packed stages held in registers ahead of the one being converted
constexpr int kL2Ahead = 8;   // stages by which the L2 prefetch of packed weights leads the x-tile loads
constexpr int kGemmThreads = 896;
constexpr int kWarpA = 0, kWarpMma = 2, kWarpEpi0 = 4, kEpiWarps = 8, kWarpDq0 = 12;
// The dequant warps form kDqGroups groups; group i converts the k-stages i, i + kDqGroups, ...
// so a warp pays the barrier handshake once per kDqGroups stages and the groups overlap each
// other's waits.
constexpr int kDqGroups = 2;
constexpr int kDqGroupWarps = 8;
constexpr int kDqRows = kBK / (2 * kDqGroupWarps);  // k rows converted by a thread per stage
constexpr int kDqRowStep = 2;                        // distance between a thread's rows
constexpr int kDqWarpRows = 2 * kDqRows;             // a warp owns this many consecutive k rows
constexpr int kSuperRows = 8;  // m-tiles per L2 super-tile
// Published tiles a role may lag behind the publisher: the publisher leads the x loads by kL2Ahead
// stages, those lead the MMAs by the ring depth, the epilogue trails by at most two tiles; with one
// stage per tile that is kL2Ahead + kNS + 2 tiles.
static_assert(kL2Ahead + kNS + 2 < kTileRing, "a slot is read before it is written again");
constexpr int kBarrierBytes = 1024;  // shared memory reserved for GmBarriers
constexpr int kEpiScaleFloats = 2 * kBN;  // per epilogue warp: the tile's column scales and scale * offset
constexpr int kAHalfBytes = kBM * kBK * 2;   // one 128-row box
constexpr int kATileBytes = 2 * kAHalfBytes;  // an x stage holds both row halves
constexpr int kSmallRows = 32;                 // rows of the small x box (a nearly empty last row half)
constexpr int kSmallBytes = kSmallRows * kBK * 2;
// A last row half of at most this many rows is multiplied with M = 64, and its x comes in boxes of 32 rows: no less time on the tensor
// core, but half of its shared-memory reads of x, fewer x bytes from L2, and less power.  us in a steady loop, M = 128 | M = 64: 65536 rows by
// popularity over 256 experts (two thirds of them with at most 64), 7168 x 4096: int8 4773 | 4604, fp8 5428 | 5222; stored fp4, 1021 tokens x 8
// over 256 experts, 2048 x 7168: 1143 | 1069; fp4-stored layer of 4096 tokens x 8: 4575 | 4378.
constexpr int kHalfM = 64;
constexpr int kBTileBytes = kBK * kBN * 2;
constexpr uint32_t kTmemCols = 512;

// Internal kernel mode: fp4 weights in the stored ("ascend") order, read as they are.  In that order a
// 64-row x 128-byte tile of the canonical matrix is still a 64 x 128-byte box of the same 2-D array
// (row = (b*4 + a)*8 + p, 128 bytes = [q (4)][c8 (8)][4 bytes], for canonical row 16a + 8b + c8 and
// byte column 128j + 16p + 4q + s), so tensor maps and strides are those of the canonical layout
// and only the thread -> data assignment of the dequant warps changes: a thread takes 8 rows x 8
// columns (two 16-byte loads) instead of 4 rows x 16 columns.
constexpr int kCtFp4Ascend = 16;
// Internal kernel mode: canonical fp4 codes with one e8m0 scale byte per 32 columns of a k row (the format of
// b200moe_fp4_dequant), dequantised by the dequant warps to the bits that operator would write.  With SILU the
// gate columns come first in the matrix and the kernel pairs them with the up columns itself.  Against writing the
// bf16 weights to memory and reading them back (4 of 4.5 bytes per weight of such a pass, and the bound of it), a
// layer of 256 experts, 4096 tokens x 8, 7168 x 2048 takes 5.08 instead of 8.80 ms, and one of few tokens an eighth.
constexpr int kCtFp4E8m0 = 17;

// Internal kernel mode: int4 weights as f16, in one pass (see "int4 in one pass" below).
constexpr int kCtInt4F16 = 18;
constexpr int kInt4ScaleShift = 6;      // the scales enter times 2^6
constexpr int kInt4BadRows = 512;       // one row in as many that is not exact in f16: all tiles go to the two-pass kernel
constexpr int kRowNotF16 = -(1 << 30);  // in the place of a row's exponent

template <int MODE>
struct GmTraits {
    static constexpr bool kNibbles = (MODE == B200MOE_CT_FP4 || MODE == B200MOE_CT_INT4 || MODE == kCtFp4Ascend ||
                                      MODE == kCtFp4E8m0 || MODE == kCtInt4F16);
    // int4 with per-128-k scale/offset: (w + o) * s does not fit bf16, so every k block is fed to
    // the tensor core twice -- a stage carries two weight tiles, hi = bf16(v) and lo = bf16(v - hi),
    // multiplied with the same x block; the fp32 accumulator then holds x @ v to about 2^-16 relative.
    static constexpr int kParts = (MODE == B200MOE_CT_INT4) ? 2 : 1;
    // ring depth: 3 x (32 + 32 KB) or 2 x (32 + 64 KB), 192 KB either way
    static constexpr int kStages = (kParts == 1) ? kNS : 2;
    static constexpr int kPRowBytes = kNibbles ? kBN / 2 : kBN;
    static constexpr int kPTileBytes = kPRowBytes * kBK;
    // bf16 weights need no conversion: TMA writes the 64-column blocks of the weight tile straight
    // into the B ring (a 64 k x 128-byte box with the 128-byte swizzle is exactly one block of the
    // MN-major operand layout) and the dequant warps have nothing to do
    static constexpr bool kDirect = (MODE == B200MOE_CT_BF16);
    // last row halves of at most this many rows are multiplied with M = 64 (not bf16, whose B tiles never pass the warps; it is free of
    // what the M = 64 forms cost: with it, 40 bytes of spills and 5 % at every size)
    static constexpr int kShortRows = kDirect ? 0 : kHalfM;
    // a dequant thread converts 8 rows x 8 columns of a stage (one 16-byte chunk of each of its rows) instead of
    // 4 rows x 16 columns: stored-order fp4 comes that way, int4 then holds and unpacks the scales and offsets of 8
    // columns instead of 16 (222 -> 14 bytes of spills; 8192 tokens x 8 over 256 experts, 7168 x 4096: 11.3 -> 9.2 ms)
    static constexpr bool kEightRows = (MODE == kCtFp4Ascend || MODE == B200MOE_CT_INT4 || MODE == kCtInt4F16);
    // Who turns a published tile number into rows and columns: the publisher, once, or each role for itself.  Resolved
    // entries cost the roles less at a tile switch but leave the dequant loop of the modes with 4 rows x 16 columns a thread
    // fewer registers.  Each role | publisher, us, libraries called in turn: 8192 tokens x 8 by popularity over 256 experts,
    // 7168 x 4096: int8 4919 | 4992, its SiLU form 4984 | 5328, fp8 5579 | 7086, canonical fp4 5089 | 6088, bf16 5072 | 5001;
    // (in runs of their own) int4 9000 | 8616, stored fp4 4838 | 4875, fp4 with e8m0 scales 4602 | 4598, SiLU 5265 | 5039.  32 rows an
    // expert, 2048 x 7168: int8 1282 | 1299, fp8 1490 | 1921, canonical fp4 1288 | 1619, int4 2326 | 2104, stored fp4 1238 |
    // 1181, e8m0 1425 | 1159.  64 experts of 210 rows, 1280 x 512: int8 52.3 | 50.3, bf16 35.9 | 34.9, stored fp4 30.8 | 28.9.
    // int8 has both, by the length of its tiles (kInt8RolesK).
    static constexpr bool kResolved = MODE != B200MOE_CT_INT8 && MODE != B200MOE_CT_FP8 && MODE != B200MOE_CT_FP4;
};

struct GmBarriers {
    uint64_t full[kNS];   // TMA bytes of the x boxes + the dequant warps of the stage's group
    uint64_t empty[kNS];  // one tcgen05.commit per stage
    // accumulator hand-off, one pair per 256-column accumulator: a two-half tile uses both, a one-half
    // tile alternates between them so that its epilogue overlaps the next tile's main loop
    uint64_t t_full[2], t_empty[2];
    uint64_t drain;
    uint32_t tmem_base;
    int abort;
    int n_tiles;
    int pad;
    // Tile schedule of this CTA: tiles are drawn from a global ticket counter (status word 2) by the
    // thread that runs furthest ahead, resolved by it and published here (tile_ring.h), the i-th tile with number i + 1.
    // Every role walks the entries in order, so all see the same sequence, and none
    // repeats the search and the divisions at each tile switch (64 experts, 210 rows each, 1280 x 512, int4: 74 -> 48 us).
    // Where the roles resolve the tiles themselves, an entry's first word is {i + 1, tile number, ~0 past the end}.
    alignas(16) TileEntry tile_ring[kTileRing];
};

struct TileInfo {
    int g, row0, n0;
    int rows;    // of the expert inside the tile, 1 .. kTileM
    int halves;  // 1: at most 128 rows in the tile, 2: more
};

// Bounded wait on a pipeline barrier.  The fast path is a single try_wait; the slow path polls,
// notices an abort raised by another role and gives up after ptx::kWaitLimitNs.
__device__ __noinline__ bool gm_wait_slow(uint32_t bar, uint32_t parity, GmBarriers* sb, int* status, int id) {
    volatile int* abort = &sb->abort;
    const uint64_t t0 = ptx::globaltimer_ns();
    uint32_t spins = 0;
    while (!ptx::mbar_try_wait(bar, parity)) {
        if ((++spins & 0xFF) == 0) {
            if (*abort) return false;
            if (ptx::globaltimer_ns() - t0 > ptx::kWaitLimitNs) {
                *abort = 1;
                report_status(status, kDevWaitExpired, id);
                return false;
            }
        }
    }
    return true;
}
__device__ __forceinline__ bool gm_wait(uint64_t* bar, uint32_t parity, GmBarriers* sb, int* status, int id) {
    const uint32_t b = ptx::smem_u32(bar);
    if (ptx::mbar_try_wait(b, parity)) return true;
    return gm_wait_slow(b, parity, sb, status, id);
}

// Waits for slot `e` to hold the tile numbered `want`; an entry of no rows when a wait expired or another role aborted.
__device__ __noinline__ TileEntry ring_wait(const TileEntry* e, uint32_t want, GmBarriers* sb, int* status) {
    volatile int* abort = &sb->abort;
    const uint64_t t0 = ptx::globaltimer_ns();
    uint32_t spins = 0;
    TileEntry v;
    while (!tile_entry_is(v = ring_load(e), want)) {
        if ((++spins & 0xFF) == 0) {
            if (*abort) return tile_entry(want, 0u, 0u, 0u, 0u);
            if (ptx::globaltimer_ns() - t0 > ptx::kWaitLimitNs) {
                *abort = 1;
                report_status(status, kDevWaitExpired, 90);
                return tile_entry(want, 0u, 0u, 0u, 0u);
            }
        }
    }
    return v;
}

// tile index -> expert, first row, rows, first column.
// Tile numbering: first every tile with two row halves (more than 128 rows), expert by expert in
// super-tiles, then every tile with one row half (the last, short m-tile of an expert).  tile_prefix
// holds two prefix arrays of G + 1 entries each: two-half tiles before expert g, one-half tiles
// before expert g.
__device__ __forceinline__ TileInfo locate_tile(int t, const int* tile_prefix, const int* row_start, int G, int n_nt) {
    const int n_two = tile_prefix[G];
    const bool two = t < n_two;
    const int* pref = two ? tile_prefix : tile_prefix + (G + 1);
    const int tt = two ? t : t - n_two;
    int lo = 0, hi = G;  // largest g with pref[g] <= tt
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pref[mid] <= tt) lo = mid;
        else hi = mid;
    }
    const int g = lo;
    const int j = tt - pref[g];
    const int r0 = row_start[g], r1 = row_start[g + 1];
    TileInfo ti;
    ti.g = g;
    if (two) {
        const int mt = (pref[g + 1] - pref[g]) / n_nt;
        // super-tiles of up to kSuperRows m-tiles x all n-tiles keep x rows and the expert's weights
        // L2-resident while they are shared by concurrently running CTAs
        const int per_super = kSuperRows * n_nt;
        const int st = j / per_super;
        const int base = st * kSuperRows;
        const int h = min(kSuperRows, mt - base);
        const int jj = j - st * per_super;
        ti.n0 = (jj / h) * kBN;
        ti.row0 = r0 + (base + jj % h) * kTileM;
        ti.halves = 2;
    } else {
        ti.n0 = j * kBN;
        ti.row0 = r0 + ((r1 - r0) / kTileM) * kTileM;
        ti.halves = 1;
    }
    ti.rows = min(r1 - ti.row0, kTileM);
    return ti;
}

// The seq-th tile of this CTA (seq counts from 0 and is advanced) into `ti`; false when the schedule has
// ended, a wait expired or another role aborted.  The publisher is always far ahead, so outside the
// first microseconds of the kernel the entry is already there.
template <bool RESOLVED>
__device__ __forceinline__ bool next_tile(GmBarriers* sb, uint32_t& seq, TileInfo& ti, const int* tile_prefix, const int* row_start,
                                          int G, int n_nt, int* status) {
    const TileEntry* e = &sb->tile_ring[seq % kTileRing];
    if constexpr (!RESOLVED) {
        const volatile uint64_t* e2 = &e->a;
        const uint32_t want = seq + 1;
        uint64_t v = *e2;
        if ((uint32_t)v != want) {
            volatile int* abort = &sb->abort;
            const uint64_t t0 = ptx::globaltimer_ns();
            uint32_t spins = 0;
            while ((uint32_t)(v = *e2) != want) {
                if ((++spins & 0xFF) == 0) {
                    if (*abort) return false;
                    if (ptx::globaltimer_ns() - t0 > ptx::kWaitLimitNs) {
                        *abort = 1;
                        report_status(status, kDevWaitExpired, 90);
                        return false;
                    }
                }
            }
        }
        ++seq;
        const uint32_t t = (uint32_t)(v >> 32);
        if (t == ~0u) return false;
        ti = locate_tile((int)t, tile_prefix, row_start, G, n_nt);
        return true;
    }
    TileEntry v = ring_load(e);
    if (!tile_entry_is(v, seq + 1)) v = ring_wait(e, seq + 1, sb, status);
    ++seq;
    ti.row0 = tile_entry_row0(v);
    ti.g = tile_entry_expert(v);
    ti.rows = tile_entry_rows(v);
    ti.n0 = tile_entry_column(v) * kBN;
    ti.halves = ti.rows > kBM ? 2 : 1;
    return ti.rows != 0;
}

// Row boundaries and the tile-count prefixes of locate_tile, by the whole CTA (a barrier must follow).  Not inlined:
// the main loops then keep their registers (inlined, every mode spilled more; int8, 8192 tokens x 8 over 256
// experts, 7168 x 4096: 5.22 -> 5.03 ms).
__device__ __noinline__ void gm_schedule(const int64_t* __restrict__ gl, int G, int M, int gl_type, int n_nt,
                                         int* row_start, int* tile_prefix, int* n_tiles, int* status) {
    load_row_starts(gl, G, M, gl_type, row_start, status);
    if (threadIdx.x < 32) {
        // tile-count prefixes, each lane over a stretch of consecutive experts
        int* pref1 = tile_prefix + (G + 1);
        int lo, hi, c2 = 0, c1 = 0, t2, t1;
        lane_experts(G, lo, hi);
        for (int g = lo; g < hi; ++g) {
            const int rows = row_start[g + 1] - row_start[g], tail = rows % kTileM;
            c2 += rows / kTileM + (tail > kBM ? 1 : 0);   // m-tiles with two row halves
            c1 += (tail >= 1 && tail <= kBM) ? 1 : 0;      // the short last m-tile, if any
        }
        int p2 = warp_exclusive_sum(c2, t2), p1 = warp_exclusive_sum(c1, t1);
        for (int g = lo; g < hi; ++g) {
            const int rows = row_start[g + 1] - row_start[g], tail = rows % kTileM;
            tile_prefix[g] = p2 * n_nt;
            pref1[g] = p1 * n_nt;
            p2 += rows / kTileM + (tail > kBM ? 1 : 0);
            p1 += (tail >= 1 && tail <= kBM) ? 1 : 0;
        }
        if (threadIdx.x == 0) {
            tile_prefix[G] = t2 * n_nt;
            pref1[G] = t1 * n_nt;
            *n_tiles = (t2 + t1) * n_nt;
        }
    }
}

// ---- dequant of one packed stage into the bf16 UMMA tile --------------------------------------
// bf16 tile layout (MN-major, 128-byte swizzle): four blocks of 64 columns; inside a block row k
// occupies 128 bytes at k*128 and its eight 16-byte chunks are XOR-swizzled with (k & 7).
__device__ __forceinline__ uint32_t btile_offset(int k, int nchunk16) {  // nchunk16: 16-byte chunk 0..31
    return (uint32_t)((nchunk16 >> 3) * (kBK * 128) + k * 128 + (((nchunk16 & 7) ^ (k & 7)) << 4));
}

// Thread -> (row, 16-column chunk) assignment of the dequant warps.  A warp owns kDqWarpRows
// consecutive k rows (inside one 16-row scale group of the fp4 format) and converts them two at a
// time (an even one and the next).  Each quarter-warp holds four lanes on the even row in
// 64-column block p and four lanes on the odd row in block p^1: the 128-bit stores of a quarter
// then hit eight different 16-byte bank groups (the swizzle term k&7 differs in its low bit
// between the two rows), and the packed loads of a warp still cover both rows contiguously.
struct DqLane {
    int row;  // the thread converts k = row + kDqRowStep * j, j < kDqRows, of its stages
    int c16;  // 16-column chunk 0..15
    // kEightRows only: the thread converts canonical rows k0 .. k0 + 7, columns 8 * chunk .. + 7
    int k0, chunk, src_row, src_byte;  // where its first bytes are inside the 64 x 128-byte box
};
template <int MODE>
__device__ __forceinline__ DqLane dq_lane(int tid) {
    const int w = tid >> 5, l = tid & 31;
    DqLane d;
    if constexpr (MODE == kCtFp4Ascend) {
        const int a = w >> 1, b = w & 1;      // warp <-> rows 16a + 8b .. + 7 (one 16-row scale group)
        d.k0 = 16 * a + 8 * b;
        d.chunk = l;                          // lane <-> 16-byte chunk of the bf16 tile row (8 columns)
        d.src_row = (b * 4 + a) * 8 + (l >> 2);
        d.src_byte = (l & 3) * 32;
        d.row = d.src_row;                    // what dq_locate adds to the stage's first row
        d.c16 = 0;
    } else if constexpr (GmTraits<MODE>::kEightRows) {
        d.k0 = d.row = d.src_row = 8 * w;
        d.chunk = l;
        d.src_byte = 4 * l;
        d.c16 = 0;
    } else {
        const int p = l >> 3, q = l & 7, odd = q >> 2;
        d.row = kDqWarpRows * w + odd;
        d.c16 = 4 * (p ^ odd) + (q & 3);
        d.k0 = d.chunk = d.src_row = d.src_byte = 0;
    }
    return d;
}

// Packed weights of one stage held by a thread: kDqRows rows x 16 columns.
template <int MODE>
struct PackedRegs {
    uint4 q[kDqRows];  // fp4 / int4 use only .x/.y of each
    uint4 s[2];        // fp4 only: the bf16 scales of the thread's 16 columns (one 16-row group)
    uint32_t e[kDqRows];  // fp4 with e8m0 scales: the scale byte of each of the thread's rows; int4: e[0] locates its scales
    float sf;          // fp8 only: the fp32 scale of the thread's 128 x 128 block
};

// Position of a dequant thread in the (tile, k-stage) sequence of its CTA, with the address of the
// thread's first packed row of that stage carried along (advanced by a constant inside a tile).
struct DqIter {
    int kt, g, n0;
    uint32_t seq;  // tiles taken from the CTA's schedule so far
    bool valid;
    const uint8_t* wp;
};
// First weight column of 16-column chunk c16 of the tile at n0.  SPLIT: the tile's lower half is the gate
// columns n0 / 2 .. + 127 and its upper half the up columns N / 2 + the same indices.
template <bool SPLIT>
__device__ __forceinline__ int chunk_col(int n0, int c16, int N) {
    return SPLIT ? (n0 >> 1) + (c16 & 7) * 16 + (c16 >> 3) * (N >> 1) : n0 + c16 * 16;
}
template <int MODE, bool SPLIT>
__device__ __forceinline__ void dq_locate(DqIter& it, const uint8_t* __restrict__ w, const GemmArgs& a, const DqLane& d) {
    using T = GmTraits<MODE>;
    if (!it.valid) return;
    const size_t row_bytes = T::kNibbles ? (size_t)a.N / 2 : (size_t)a.N;
    it.wp = w + ((size_t)it.g * a.K + (size_t)it.kt * kBK + d.row) * row_bytes +
            (T::kEightRows        ? (it.n0 >> 1) + d.src_byte
             : T::kNibbles        ? chunk_col<SPLIT>(it.n0, d.c16, a.N) >> 1
                                  : it.n0 + d.c16 * 16);
}
template <int MODE, bool SPLIT, bool RESOLVED>
__device__ __forceinline__ void dq_advance(DqIter& it, int step, const uint8_t* __restrict__ w, const GemmArgs& a,
                                           const DqLane& d, int n_kt, const int* tile_prefix, const int* row_start, int n_nt, GmBarriers* sb) {
    using T = GmTraits<MODE>;
    it.kt += step;
    if (it.kt < n_kt) {
        it.wp += (size_t)step * kBK * (T::kNibbles ? (size_t)a.N / 2 : (size_t)a.N);
        return;
    }
    do {
        it.kt -= n_kt;
        TileInfo ti;
        it.valid = next_tile<RESOLVED>(sb, it.seq, ti, tile_prefix, row_start, a.G, n_nt, a.status);
        it.g = ti.g;
        it.n0 = ti.n0;
    } while (it.kt >= n_kt && it.valid);
    dq_locate<MODE, SPLIT>(it, w, a, d);
}

constexpr int kScaleAhead = 6;  // stages by which the e8m0 scale lines are requested into L2

template <int MODE, bool SPLIT>
__device__ __forceinline__ void load_packed(PackedRegs<MODE>& r, const DqIter& it, const GemmArgs& a, const DqLane& d) {
    using T = GmTraits<MODE>;
    if constexpr (MODE == kCtFp4Ascend) {
        // 32 consecutive bytes = rows c8 = 0..7 of the thread's 8 columns, 4 bytes each; one scale
        // vector (8 columns of the rows' 16-row group)
        r.q[0] = __ldg(reinterpret_cast<const uint4*>(it.wp));
        r.q[1] = __ldg(reinterpret_cast<const uint4*>(it.wp + 16));
        r.s[0] = __ldg(reinterpret_cast<const uint4*>(
            static_cast<const __nv_bfloat16*>(a.scale) +
            ((size_t)it.g * (a.K >> 4) + ((it.kt * kBK + d.k0) >> 4)) * a.N + it.n0 + d.chunk * 8));
        return;
    }
    const size_t row_bytes = T::kNibbles ? (size_t)a.N / 2 : (size_t)a.N;
    if constexpr (MODE == B200MOE_CT_INT4 || MODE == kCtInt4F16) {
        uint32_t v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = ldg_stream4(it.wp + (size_t)i * row_bytes);
        r.q[0] = make_uint4(v[0], v[1], v[2], v[3]);
        r.q[1] = make_uint4(v[4], v[5], v[6], v[7]);
        // in units of the 8 scales a thread loads (fits 32 bits: 2^32 of them are the scales of 2.2 TB of weights)
        r.e[0] = (uint32_t)((((size_t)it.g * (a.K >> 7) + ((it.kt * kBK) >> 7)) * a.N + it.n0) >> 3) + d.chunk;
        return;
    }
#pragma unroll
    for (int j = 0; j < kDqRows; ++j) {
        const uint8_t* p = it.wp + (size_t)(kDqRowStep * j) * row_bytes;
        if constexpr (T::kNibbles) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
            r.q[j] = make_uint4(v.x, v.y, 0u, 0u);
        } else if (MODE != B200MOE_CT_FP8 || it.n0 + d.c16 * 16 < a.N) {
            r.q[j] = MODE == B200MOE_CT_FP8 ? ldg_stream(p) : __ldg(reinterpret_cast<const uint4*>(p));
        } else {
            r.q[j] = make_uint4(0u, 0u, 0u, 0u);  // columns past N in the 128-column last tile of an fp8 matrix
        }
    }
    if constexpr (MODE == B200MOE_CT_FP8) {
        r.sf = it.n0 + d.c16 * 16 < a.N
                   ? __ldg(static_cast<const float*>(a.scale) + ((size_t)it.g * (a.K >> 7) + ((it.kt * kBK) >> 7)) * (a.N >> 7) +
                           ((it.n0 + d.c16 * 16) >> 7))
                   : 0.f;
    }
    if constexpr (MODE == kCtFp4E8m0) {
        const uint8_t* sc = static_cast<const uint8_t*>(a.scale);
        const size_t ld = (size_t)a.N >> 5, row0 = (size_t)it.g * a.K + (size_t)it.kt * kBK;
        const uint8_t* sp = sc + (row0 + d.row) * ld + (chunk_col<SPLIT>(it.n0, d.c16, a.N) >> 5);
#pragma unroll
        for (int j = 0; j < kDqRows; ++j) r.e[j] = __ldg(sp + (size_t)(kDqRowStep * j) * ld);
        // a tile's scales are 8 bytes of a k row's line: the lines of the warp's eight rows of a later stage are
        // requested into L2 here (SPLIT: lanes 8 .. 15 those of the up columns)
        const int l = threadIdx.x & 31, w0 = d.row & ~(kDqWarpRows - 1);
        if (l < (SPLIT ? 16 : 8) && (it.kt + kScaleAhead + 1) * kBK <= a.K)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(sc + (row0 + (size_t)kScaleAhead * kBK + w0 + (l & 7)) * ld +
                                                          (chunk_col<SPLIT>(it.n0, l & 8, a.N) >> 5)));
    }
    if constexpr (MODE == B200MOE_CT_FP4) {
        const uint4* sp = reinterpret_cast<const uint4*>(
            static_cast<const __nv_bfloat16*>(a.scale) +
            ((size_t)it.g * (a.K >> 4) + ((it.kt * kBK + d.row) >> 4)) * a.N + it.n0 + d.c16 * 16);
        r.s[0] = __ldg(sp);
        r.s[1] = __ldg(sp + 1);
    }
}

// 16-byte shared-memory store at a 32-bit shared address.
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// Shared address of the thread's chunk pair in its row j, from the address `sa` of the pair in its
// row 0: the thread's rows are k = row0 + 2j with row0 & 7 in {0, 1}, so the swizzle term changes by
// XOR with 2j (bits 5..6 of the address) and the row offset by j * 256 bytes.  The second chunk of
// the pair is at the returned address ^ 16.
__device__ __forceinline__ uint32_t dq_row_addr(uint32_t sa, int j) { return (sa ^ (uint32_t)(j << 5)) + (uint32_t)(j * 256); }

// Stored-order fp4 and fp4 with e8m0 scales enter the tile in the column order (0,4,1,5,2,6,3,7) of every eight, the order
// in which the decode produces them (e2m1x8_to_bf16_tiny); the epilogue undoes it when it picks accumulator
// registers.  Restoring the order here cost four permutes per eight codes (with resolved tiles, fp4-stored layer of 256
// experts, 4096 tokens x 8, 7168 x 2048: 4.79 -> 4.61 ms).  The scales of eight columns are
// brought into the same order, once for all rows of the scale group (the canonical order's 16 columns a thread
// leave no registers for that).
__device__ __forceinline__ uint4 pair_scales(const uint4& s) {
    return make_uint4(prmt(s.x, s.z, 0x5410u), prmt(s.x, s.z, 0x7632u), prmt(s.y, s.w, 0x5410u), prmt(s.y, s.w, 0x7632u));
}

// Whether the 2^126 that e2m1x8_to_bf16_tiny leaves out fits into the whole warp's scales (magnitudes below 4; no infinity or
// NaN): the product of the scaled scale and the tiny code is then the one rounding of code * scale.
__device__ __forceinline__ bool scales_take_2p126(const uint4& s) {
    constexpr uint32_t kMag = 0x7FFF7FFFu, kUp = 0x3F803F80u;  // 0x4080 is the bf16 4.0: + 0x3F80 carries into bit 15
    const uint32_t big = ((s.x & kMag) + kUp) | ((s.y & kMag) + kUp) | ((s.z & kMag) + kUp) | ((s.w & kMag) + kUp);
    return __all_sync(0xffffffffu, (big & 0x80008000u) == 0u);
}

// Stored-order fp4: eight rows of eight columns; `sa` is the shared address of the thread's chunk in
// its first row (a multiple of 8, so row i flips the chunk's swizzle bits by i and adds i * 128).
__device__ __forceinline__ void convert_stage_fp4_ascend(const PackedRegs<kCtFp4Ascend>& r, uint32_t sa) {
    uint4 sc = pair_scales(r.s[0]);
    const bool tiny = scales_take_2p126(sc);
    if (tiny) sc = make_uint4(mul_bf16x2(sc.x, kTwo126), mul_bf16x2(sc.y, kTwo126), mul_bf16x2(sc.z, kTwo126), mul_bf16x2(sc.w, kTwo126));
    const uint32_t w8[8] = {r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w, r.q[1].x, r.q[1].y, r.q[1].z, r.q[1].w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint32_t v[4];
        e2m1x8_to_bf16_tiny(w8[i], v);
        if (!tiny) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = mul_bf16x2(v[j], kTwo126);
        }
        sts128((sa ^ (uint32_t)(i << 4)) + (uint32_t)(i * 128), mul_bf16x2(v[0], sc.x), mul_bf16x2(v[1], sc.y),
               mul_bf16x2(v[2], sc.z), mul_bf16x2(v[3], sc.w));
    }
}

// fp8: the weight of a code c is bf16(fp32(c * s)) with the fp32 scale s of its 128 x 128 block.  Widening every code to fp32,
// multiplying and rounding takes 15 instructions per four; in bf16, fma(c, hi, c * lo) with hi + lo = s to 2^-17 takes 11 (65536
// rows over 256 experts, 7168 x 4096: 6153 -> 5908 us), and
// differs only where c * s lies that close to the middle of two bf16 numbers.  A code has one of eight significands (a subnormal
// one too), and the rounding of c * s * 2^e does not depend on e, so the eight significands tell whether a scale has such a
// code: about 1 % do and take the long way.  The block's 16 lanes of the warp try them, two lanes each.  The 2^120 of the
// codes' placement rides in hi and lo, so |s| < 128; from 2^-90 on nothing on the way is subnormal.  A zero scale is fine.
struct Fp8Scale {
    uint32_t hi, lo;  // bf16x2, both halves alike
    bool two_terms;   // for the whole warp
};
__device__ __forceinline__ Fp8Scale fp8_scale(float s) {
    Fp8Scale f;
    const float up = s * 1.329227995784916e36f;  // 2^120
    f.hi = pack_bf16x2(up, up);
    const float rest = up - __uint_as_float(f.hi << 16);
    f.lo = pack_bf16x2(rest, rest);
    const int l = threadIdx.x & 31;  // the block is the upper bit of (l >> 3) ^ (l >> 2 & 1) (dq_lane)
    const uint32_t c = 0x0380u | (uint32_t)((((l >> 3) ^ (l >> 2)) & 1) * 64 + (l & 3) * 16);  // 1.m * 2^-120
    const float full = __uint_as_float(c << 16) * up;
    const uint32_t exact = pack_bf16x2(full, 0.f), two = fma_bf16x2(c, f.hi, mul_bf16x2(c, f.lo));
    const bool in_range = fabsf(s) < 128.f && (fabsf(s) >= 8.077935669463161e-28f || s == 0.f);  // 2^-90
    f.two_terms = __all_sync(0xffffffffu, in_range && (two & 0xFFFFu) == (exact & 0xFFFFu));
    return f;
}

template <int MODE>
__device__ __forceinline__ void convert_stage(const PackedRegs<MODE>& r, uint32_t sa) {
    Fp8Scale f8;
    if constexpr (MODE == B200MOE_CT_FP8) f8 = fp8_scale(r.sf);
    bool tiny = false;
    if constexpr (MODE == kCtFp4E8m0) {
        // 2^(s - 127) * 2^126 = 2^(s - 1) is a bf16 up to s = 128 (s = 0 included: 2^-127 is a subnormal, 2^-1 is not)
        tiny = __all_sync(0xffffffffu, max(max(r.e[0], r.e[1]), max(r.e[2], r.e[3])) <= 128u);
    }
    static_assert(kDqRows == 4, "scale bytes of a thread");
#pragma unroll
    for (int j = 0; j < kDqRows; ++j) {
        const uint4 q = r.q[j];
        uint32_t o[8];
        if constexpr (MODE == B200MOE_CT_INT8) {
            // tile columns 4i..4i+3 hold weight columns 4i, 4i+2, 4i+1, 4i+3 (undone in the epilogue)
            s8x4_to_bf16_even_odd(q.x, o[0], o[1]);
            s8x4_to_bf16_even_odd(q.y, o[2], o[3]);
            s8x4_to_bf16_even_odd(q.z, o[4], o[5]);
            s8x4_to_bf16_even_odd(q.w, o[6], o[7]);
        } else if constexpr (MODE == B200MOE_CT_FP8) {
            // e4m3 byte -> bf16 with the 4 exponent and 3 mantissa bits placed under the bf16 exponent (the value
            // times 2^-120, subnormals included), bytes 0, 2 and 1, 3 of a word at a time (tile columns as for int8)
            const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                o[2 * i] = ((w4[i] << 4) & 0x07F007F0u) | ((w4[i] << 8) & 0x80008000u);
                o[2 * i + 1] = ((w4[i] >> 4) & 0x07F007F0u) | (w4[i] & 0x80008000u);
            }
            if (f8.two_terms) {
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = fma_bf16x2(o[i], f8.hi, mul_bf16x2(o[i], f8.lo));
            } else {
                const float sf = r.sf;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t v = mul_bf16x2(o[i], 0x7B807B80u);  // * 2^120
                    o[i] = pack_bf16x2(__uint_as_float(v << 16) * sf, __uint_as_float(v & 0xFFFF0000u) * sf);
                }
            }
        } else if constexpr (MODE == kCtFp4E8m0) {
            // 2^(s-127) as bf16: exponent field s; s = 0 is the subnormal 2^-127, 255 is NaN
            const uint32_t e = r.e[j];
            const uint32_t sb = tiny ? (e + 126u) * 0x800080u : (e == 0 ? 0x0040u : (e == 255 ? 0x7FC0u : (e << 7))) * 0x10001u;
            e2m1x8_to_bf16_tiny(q.x, o);
            e2m1x8_to_bf16_tiny(q.y, o + 4);
            if (!tiny) {
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = mul_bf16x2(o[i], kTwo126);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = mul_bf16x2(o[i], sb);
        } else {  // FP4: 8 bytes = 16 codes; the thread's rows share one 16-row scale group
            const uint4 s0 = r.s[0], s1 = r.s[1];
            uint32_t v[4];
            e2m1x8_to_bf16(q.x, v);
            o[0] = mul_bf16x2(v[0], s0.x); o[1] = mul_bf16x2(v[1], s0.y);
            o[2] = mul_bf16x2(v[2], s0.z); o[3] = mul_bf16x2(v[3], s0.w);
            e2m1x8_to_bf16(q.y, v);
            o[4] = mul_bf16x2(v[0], s1.x); o[5] = mul_bf16x2(v[1], s1.y);
            o[6] = mul_bf16x2(v[2], s1.z); o[7] = mul_bf16x2(v[3], s1.w);
        }
        const uint32_t aj = dq_row_addr(sa, j);
        sts128(aj, o[0], o[1], o[2], o[3]);
        sts128(aj ^ 16u, o[4], o[5], o[6], o[7]);
    }
}

// int4 with per-128-k scale / offset: one pass over a k block produces both stages it feeds to the
// tensor core, hi = bf16(v) and lo = bf16(v - hi) with v = w * s + o * s in fp32.  The thread's
// rows lie in the same 128-k group, so its 8 scales and offsets are loaded once per k block
// (before the wait for the stage, so that their latency is hidden by it).
struct Int4Scales {
    uint4 s, o;
};
__device__ __forceinline__ Int4Scales load_int4_scales(const GemmArgs& a, uint32_t unit) {
    Int4Scales r;
    r.s = __ldg(static_cast<const uint4*>(a.scale) + unit);
    r.o = a.offset != nullptr ? __ldg(reinterpret_cast<const uint4*>(a.offset) + unit) : make_uint4(0u, 0u, 0u, 0u);
    return r;
}

// `sa_hi` / `sa_lo`: shared addresses of the thread's chunk in its first row (a multiple of 8, see
// convert_stage_fp4_ascend).
__device__ __forceinline__ void convert_block_int4(const PackedRegs<B200MOE_CT_INT4>& r, const Int4Scales& sc,
                                                   uint32_t sa_hi, uint32_t sa_lo) {
    const f32x2 kMagic = pack_f32x2(8388616.0f, 8388616.0f);  // 2^23 + 8
    const uint32_t sw[4] = {sc.s.x, sc.s.y, sc.s.z, sc.s.w};
    const uint32_t ow[4] = {sc.o.x, sc.o.y, sc.o.z, sc.o.w};
    f32x2 s2[4], t2[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        s2[i] = pack_f32x2(__uint_as_float(sw[i] << 16), __uint_as_float(sw[i] & 0xFFFF0000u));
        t2[i] = mul_f32x2(pack_f32x2(__uint_as_float(ow[i] << 16), __uint_as_float(ow[i] & 0xFFFF0000u)), s2[i]);
    }
    const uint32_t w8[8] = {r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w, r.q[1].x, r.q[1].y, r.q[1].z, r.q[1].w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint32_t word = w8[j] ^ 0x88888888u;                                      // nibble + 8, unsigned
        const uint32_t lo_n = word & 0x0F0F0F0Fu, hi_n = (word >> 4) & 0x0F0F0F0Fu;  // even / odd columns, one per byte
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // column pair 2i, 2i + 1 = byte i of the word
            // byte i under the fp32 pattern of 2^23: the float 2^23 + nibble + 8
            const f32x2 wm = pack_u32x2(prmt(lo_n, 0x4B000000u, 0x7440u + i), prmt(hi_n, 0x4B000000u, 0x7440u + i));
            const f32x2 v = fma_f32x2(sub_f32x2(wm, kMagic), s2[i], t2[i]);
            hi[i] = pack_bf16x2(f32x2_lo(v), f32x2_hi(v));
            const f32x2 l = sub_f32x2(v, pack_u32x2(hi[i] << 16, hi[i] & 0xFFFF0000u));
            lo[i] = pack_bf16x2(f32x2_lo(l), f32x2_hi(l));
        }
        const uint32_t at = (uint32_t)(j << 4), row = (uint32_t)(j * 128);
        sts128((sa_hi ^ at) + row, hi[0], hi[1], hi[2], hi[3]);
        sts128((sa_lo ^ at) + row, lo[0], lo[1], lo[2], lo[3]);
    }
}

// ---- int4 in one pass --------------------------------------------------------------------------------------
// For calls without offsets.  w * s has at most 11 significant bits, which one f16 tile holds where bf16 takes a pair of tiles, and f16
// times f16 runs at the rate of bf16.  So x is written as f16 first (gm_int4_prepare_x_kernel: each row times the power of two that puts
// its largest element into [2^14, 2^15)) and the weights enter as w * s * 2^6, exact for scales of 2^-23 up to 2^7; the epilogue
// multiplies by the row's power of two.  Against the hi + lo pair of tiles: half the MMAs, 13 instead of 34 instructions per eight codes.
// Every product is exact and the accumulator takes half as many, so the fp32 sums are the closer ones (16 experts of 40 rows, 7168 x 2048,
// error against 64 bits: 0.7e-5 .. 0.8e-5, the pair of tiles 1.3e-5 .. 1.6e-5).
// With an offset (w + o) * s has up to 16 bits, which f16 does not hold, and w * s and o * s as separate products cancel where the offset does
// what a zero point is for: sums of both signs, each many times the result, in an accumulator that drops what lies 24 bits
// below it (codes with zero points, positive x: 1.0e-4 .. 3.2e-4 against 1.1e-5; codes 5 .. 7 under offsets about -6, positive x: 1.4e-2
// against 1.5e-5).  Such calls take the pair.
// Rows of x that f16 cannot hold (an element more than about 2^-32 below the row's largest, infinities, NaN) and tiles with a scale
// out of range are done again by the two-pass kernel: the epilogue lists such tiles.  Where more than
// one row in kInt4BadRows is of that kind, the two-pass kernel does all tiles and this one none.

// Whether f16 holds w * s * 2^6 for every code (two bf16 scales a word).
__device__ __forceinline__ bool int4_scale_fits(uint32_t w) {
    const uint32_t a = w & 0x7FFFu, b = (w >> 16) & 0x7FFFu;  // 0x3400: 2^-23, 0x4300: 2^7
    return (a == 0u || a - 0x3400u < 0x0F00u) && (b == 0u || b - 0x3400u < 0x0F00u);
}

// Eight rows of eight columns, in the column order of the fp4 modes; `sa` as in convert_stage_fp4_ascend.
__device__ __forceinline__ void convert_int4_f16(const PackedRegs<kCtInt4F16>& r, const uint4& s8, uint32_t sa) {
    const uint4 sp = pair_scales(s8);
    const uint32_t sb[4] = {sp.x, sp.y, sp.z, sp.w};
    __half2 sc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const f32x2 up = mul_f32x2(pack_u32x2(sb[i] << 16, sb[i] & 0xFFFF0000u), pack_f32x2(1 << kInt4ScaleShift, 1 << kInt4ScaleShift));
        sc[i] = __floats2half2_rn(f32x2_lo(up), f32x2_hi(up));
    }
    // code ^ 8 under the f16 1024 (or, four bits up, sixteen times it): one add or multiply-add gives the code's value
    const __half2 k1032 = __float2half2_rn(-1032.f), k16th = __float2half2_rn(0.0625f), k72 = __float2half2_rn(-72.f);
    const uint32_t w8[8] = {r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w, r.q[1].x, r.q[1].y, r.q[1].z, r.q[1].w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        uint32_t o[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t w = h ? w8[j] >> 8 : w8[j];
            uint32_t lo, hi;
            asm("lop3.b32 %0, %1, 0x000F000F, 0x64086408, 0x6A;" : "=r"(lo) : "r"(w));  // (w & m) ^ c
            asm("lop3.b32 %0, %1, 0x00F000F0, 0x64806480, 0x6A;" : "=r"(hi) : "r"(w));
            const __half2 v0 = __hmul2(__hadd2(*reinterpret_cast<__half2*>(&lo), k1032), sc[2 * h]);
            const __half2 v1 = __hmul2(__hfma2(*reinterpret_cast<__half2*>(&hi), k16th, k72), sc[2 * h + 1]);
            o[2 * h] = *reinterpret_cast<const uint32_t*>(&v0);
            o[2 * h + 1] = *reinterpret_cast<const uint32_t*>(&v1);
        }
        sts128((sa ^ (uint32_t)(j << 4)) + (uint32_t)(j * 128), o[0], o[1], o[2], o[3]);
    }
}

// Position of the x producer's L2 prefetch in the (tile, k-stage) sequence of its CTA.
struct StageIter {
    int kt;
    TileInfo ti;
    bool valid;
};

// Accumulator position of output column i: the int8 and fp8 dequant stores columns (0,2,1,3) of every four, the fp4 ones
// named there (0,4,1,5,2,6,3,7) of every eight.
template <int MODE>
__device__ __forceinline__ constexpr int acc_pos(int i) {
    return MODE == B200MOE_CT_INT8 || MODE == B200MOE_CT_FP8 ? ((i & ~3) | ((i & 1) << 1) | ((i >> 1) & 1))
           : (MODE == kCtFp4Ascend || MODE == kCtFp4E8m0 || MODE == kCtInt4F16) ? ((i & ~7) | ((i & 3) << 1) | ((i >> 2) & 1))
                                                            : i;
}

// One-pass int4: 2^(e - 6) of a row, and the check of a tile by one warp; what does not fit is listed for the two-pass kernel.
__device__ __forceinline__ float int4_row_unit(int e) {
    return e == kRowNotF16 ? 0.f : __uint_as_float((uint32_t)(e - kInt4ScaleShift + 127) << 23);
}
__device__ __noinline__ void int4_check_tile(const int* __restrict__ row_exp, const uint4* __restrict__ scale, int n_g, int stride, int g, int row0, int rows, int n0, int4* redo, int* redo_count) {
    const int lane = threadIdx.x & 31;
    bool ok = true;
    for (int i = lane; i < rows; i += 32) ok = ok && __ldca(row_exp + row0 + i) != kRowNotF16;
    const size_t first = (size_t)g * n_g * stride + (n0 >> 3) + lane;
#pragma unroll 4
    for (int i = 0; i < n_g; ++i) {
        const uint4 s = __ldg(scale + first + (size_t)i * stride);
        ok = ok && int4_scale_fits(s.x) && int4_scale_fits(s.y) && int4_scale_fits(s.z) && int4_scale_fits(s.w);
    }
    if (!__all_sync(0xffffffffu, ok) && lane == 0) redo[atomicAdd(redo_count, 1)] = make_int4(g, row0, rows, n0);
}

// SILU (int8, fp4 with e8m0 scales): int8 weight columns come as blocks of 128 gate columns followed by the 128
// up columns of the same indices (fp4: gate columns first, paired here), and the epilogue writes bf16(silu(gate) * up), [M, N/2], instead of
// the [M, N] product (gate and up are rounded to bf16 first, as the unfused operators would).
template <int MODE, bool SILU, bool RESOLVED>
__global__ void __launch_bounds__(kGemmThreads, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_xs,
                    const __grid_constant__ CUtensorMap tmap_w, const uint8_t* __restrict__ weight, const GemmArgs a) {
    using T = GmTraits<MODE>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* a_ring = base;
    constexpr int NS = T::kStages, P = T::kParts;
    constexpr bool SPLIT = SILU && MODE == kCtFp4E8m0;
    uint8_t* b_ring = a_ring + NS * kATileBytes;
    GmBarriers* sb = reinterpret_cast<GmBarriers*>(b_ring + NS * P * kBTileBytes);
    static_assert(sizeof(GmBarriers) <= kBarrierBytes, "barrier block");
    float* epi_scale = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(sb) + kBarrierBytes);
    int* row_start = reinterpret_cast<int*>(epi_scale + kEpiWarps * kEpiScaleFloats);
    int* tile_prefix = row_start + (a.G + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_nt = (a.N + kBN - 1) / kBN;  // (fp8 only: the last tile may hold 128 columns)
    const int n_kt = a.K / kBK;  // stages per tile

    if constexpr (MODE == B200MOE_CT_INT4) {
        if (a.redo_ctl != nullptr) {
            grid_dep_wait();
            if (__ldcg(a.redo_ctl) == 0 && __ldcg(a.redo_ctl + 2) == 0) return;  // no tile to do again
        }
    }
    gm_schedule(a.group_list, a.G, a.M, a.gl_type, n_nt, row_start, tile_prefix, &sb->n_tiles, a.status);
    if (threadIdx.x == 32) {
        sb->abort = 0;
        for (int i = 0; i < kTileRing; ++i) sb->tile_ring[i] = tile_entry(0u, 0u, 0u, 0u, 0u);
        for (int i = 0; i < NS; ++i) {
            ptx::mbar_init(ptx::smem_u32(&sb->full[i]), T::kDirect ? 1 : 1 + kDqGroupWarps);
            ptx::mbar_init(ptx::smem_u32(&sb->empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(ptx::smem_u32(&sb->t_full[i]), 1);
            ptx::mbar_init(ptx::smem_u32(&sb->t_empty[i]), kEpiWarps / 2);
        }
        ptx::mbar_init(ptx::smem_u32(&sb->drain), 1);
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tmap_x);
        ptx::prefetch_tensormap(&tmap_xs);
        ptx::prefetch_tensormap(&tmap_w);
    }
    if (warp == kWarpMma) {
        ptx::tmem_alloc(ptx::smem_u32(&sb->tmem_base), kTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();

    // (launched behind the row sums' kernel, everything up to here ran beside it: it zeroes the tile ticket)
    grid_dep_wait();

    int n_tiles = sb->n_tiles;
    bool listed = false;  // the tiles come from the list of those to do again
    if constexpr (MODE == kCtInt4F16 || MODE == B200MOE_CT_INT4) {
        if (a.redo_ctl != nullptr) {
            const bool all_again = (long long)__ldcg(a.redo_ctl + 2) * kInt4BadRows > row_start[a.G];
            if (MODE == kCtInt4F16 && all_again) n_tiles = 0;
            if (MODE == B200MOE_CT_INT4 && !all_again) {
                listed = true;
                n_tiles = __ldcg(a.redo_ctl);
            }
        }
    }
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&sb->tmem_base);

    if (warp == kWarpA) {
        // ------------------------------ x-tile producer ------------------------------
        // Also pulls the packed weight tile of the stage kL2Ahead further on into L2 (a TMA
        // prefetch has no shared-memory destination), so the dequant warps' register loads, which
        // can only run a stage or two ahead, find their data in L2 instead of waiting on HBM.
        if (lane == 0) {
            uint32_t ia = 0, seq = 0, published = 0;
            bool ok = true;
            // This thread runs furthest ahead (its L2 prefetch leads everything else), so it draws the
            // tiles.  One ticket is always held in hand, so the atomic's latency is off the path.
            // zero at the start: by a memset before the launch, or by the row sums' or x preparing kernel
            int* ticket = MODE == B200MOE_CT_INT4 && a.redo_ctl != nullptr ? a.redo_ctl + 1 : a.status + 2;
            int held = atomicAdd(ticket, 1);
            StageIter far;  // the tile published last
            far.kt = 0;
            auto publish = [&]() {
                far.valid = held < n_tiles;
                TileEntry entry = tile_entry(published + 1, RESOLVED ? 0u : ~0u, 0u, 0u, 0u);
                if (far.valid) {
                    if (MODE == B200MOE_CT_INT4 && listed) {
                        const int4 e = __ldcg(a.redo + held);
                        far.ti.g = e.x;
                        far.ti.row0 = e.y;
                        far.ti.rows = e.z;
                        far.ti.n0 = e.w;
                    } else {
                        far.ti = locate_tile(held, tile_prefix, row_start, a.G, n_nt);
                    }
                    entry = tile_entry(published + 1, (uint32_t)(RESOLVED ? far.ti.row0 : held), (uint32_t)far.ti.rows,
                                       (uint32_t)far.ti.g, (uint32_t)far.ti.n0 / kBN);
                }
                ring_store(&sb->tile_ring[published % kTileRing], entry);
                ++published;
                if (far.valid) held = atomicAdd(ticket, 1);
            };
            publish();
            auto far_step = [&]() {
                if constexpr (SPLIT) {
                    ptx::tma_prefetch_l2_2d(&tmap_w, far.ti.n0 / 4, far.ti.g * a.K + far.kt * kBK);
                    ptx::tma_prefetch_l2_2d(&tmap_w, (a.N + far.ti.n0) / 4, far.ti.g * a.K + far.kt * kBK);
                } else if constexpr (!T::kDirect)
                    ptx::tma_prefetch_l2_2d(&tmap_w, T::kNibbles ? far.ti.n0 / 2 : far.ti.n0, far.ti.g * a.K + far.kt * kBK);
                if (++far.kt < n_kt) return;
                far.kt = 0;
                publish();
            };
            for (int i = 0; i < kL2Ahead && far.valid; ++i) far_step();
            for (;;) {
                TileInfo ti;
                if (!next_tile<RESOLVED>(sb, seq, ti, tile_prefix, row_start, a.G, n_nt, a.status) || !ok) break;
                // The last row half of a tile often holds only a few rows of the expert (a second half
                // of a dozen rows when an expert has a little over 128): up to kHalfM rows come in one or two boxes of kSmallRows
                // rows.  The MMA reads kHalfM rows then; what those beyond the boxes
                // hold is left over from earlier stages and lands in accumulator rows that are never
                // stored.
                const int last_rows = ti.rows - (ti.halves - 1) * kBM;
                const int n_small = last_rows <= max(T::kShortRows, kSmallRows) ? (last_rows + kSmallRows - 1) / kSmallRows : 0;
                const uint32_t stage_bytes = (uint32_t)((ti.halves - 1) * kAHalfBytes + (n_small ? n_small * kSmallBytes : kAHalfBytes));
                const CUtensorMap* last_map = n_small ? &tmap_xs : &tmap_x;
                for (int kt = 0; kt < n_kt; ++kt, ++ia) {
                    const uint32_t s = ia % NS, ph = (ia / NS) & 1;
                    if (ia >= NS && !gm_wait(&sb->empty[s], ph ^ 1, sb, a.status, 10 + (int)s)) { ok = false; break; }
                    const uint32_t bar = ptx::smem_u32(&sb->full[s]);
                    const int kx = kt * kBK;
                    ptx::mbar_arrive_expect_tx(bar, stage_bytes + (T::kDirect ? (uint32_t)kBTileBytes : 0u));
                    if constexpr (T::kDirect) {
#pragma unroll
                        for (int blk = 0; blk < kBN / 64; ++blk)
                            ptx::tma_load_2d(ptx::smem_u32(b_ring + s * kBTileBytes + blk * (kBK * 128)), &tmap_w, bar,
                                             ti.n0 + blk * 64, ti.g * a.K + kx);
                    }
                    uint32_t dst = ptx::smem_u32(a_ring + s * kATileBytes);
                    int row = ti.row0;
                    if (ti.halves == 2) {
                        ptx::tma_load_2d(dst, &tmap_x, bar, kx, row);
                        dst += kAHalfBytes;
                        row += kBM;
                    }
                    // (no loop over the boxes: 32 experts, 264 tokens x 4, 4096 x 1024: int8 91.3 -> 80.2 us, stored fp4 51.7 -> 47.1)
                    ptx::tma_load_2d(dst, last_map, bar, kx, row);
                    if (T::kShortRows > kSmallRows && n_small == 2) ptx::tma_load_2d(dst + kSmallBytes, &tmap_xs, bar, kx, row + kSmallRows);
                    if (far.valid) far_step();
                }
            }
            if (!ok)
                for (uint32_t j = (ia > NS ? ia - NS : 0); j < ia; ++j)
                    (void)ptx::mbar_wait(ptx::smem_u32(&sb->full[j % NS]), (j / NS) & 1);
        }
    } else if (warp == kWarpMma) {
        // ------------------------------ MMA issuer ------------------------------
        // The whole warp walks the loop, so that waits, tile look-up and descriptor arithmetic are warp-uniform, and
        // one elected lane issues the tcgen05 instructions: with everything in a branch of one lane, the issue of a
        // stage's MMAs took 750 cycles, as long as they run, and stood in the ring's round trip (8192 tokens x 8 over 256
        // experts, 7168 x 4096, int8: 5.03 -> 4.90 ms; the fp4-stored layer's GEMMs 5.24 -> 5.05).  Ring positions
        // and parities are carried incrementally and the shared-memory descriptors are a 64-bit base plus a
        // small stage / k offset.  The next stage's barrier is polled (non-blocking) right after a stage's MMAs are
        // issued, so that the poll's latency runs beside the commit's.
        const bool leader = ptx::elect_one();
        const uint32_t idesc = MODE == kCtInt4F16 ? ptx::umma_idesc_f16(kBM, kBN, true) : ptx::umma_idesc_bf16(kBM, kBN, true);
        // A: K-major, 8-row groups 1024 B apart, 32 B per 16 k inside the swizzle atom
        const uint64_t da0 = ptx::umma_desc_sw128(ptx::smem_u32(a_ring), 0, 1024);
        // B: MN-major, 64-column blocks kBK*128 B apart (LBO), 8-k groups 1024 B apart (SBO)
        const uint64_t db0 = ptx::umma_desc_sw128(ptx::smem_u32(b_ring), kBK * 128, 1024);
        uint32_t sa = 0, pha = 0;
        uint32_t uses0 = 0, uses1 = 0, next1 = 0;
        bool ok = true, ready = false;  // ready: the next stage's barrier has been seen complete already
        uint32_t seq = 0;
        for (;;) {
            TileInfo ti;
            if (!__all_sync(0xffffffffu, next_tile<RESOLVED>(sb, seq, ti, tile_prefix, row_start, a.G, n_nt, a.status))) break;
            // accumulators of this tile: both for two halves, else the one used less recently;
            // the epilogue of their previous tile must have drained them
            const bool use0 = ti.halves == 2 || next1 == 0, use1 = ti.halves == 2 || next1 == 1;
            if (ti.halves == 1) next1 ^= 1u;
            if (use0 && uses0 >= 1) ok = gm_wait(&sb->t_empty[0], (uses0 - 1) & 1, sb, a.status, 30);
            if (ok && use1 && uses1 >= 1) ok = gm_wait(&sb->t_empty[1], (uses1 - 1) & 1, sb, a.status, 31);
            if (!__all_sync(0xffffffffu, ok)) break;
            const uint32_t acc0 = tmem_base + (use0 ? 0u : (uint32_t)kBN);
            // M = 64 instead of 128 in the last row half: what is taken off the instruction descriptors
            const uint32_t less = T::kShortRows > 0 && ti.rows - (ti.halves - 1) * kBM <= T::kShortRows ? (uint32_t)((kBM - kHalfM) >> 4) << 24 : 0u;
            ptx::tc_fence_after();
            uint32_t accumulate = 0;
            for (int kt = 0; kt < n_kt; ++kt) {
                if (!ready) ok = __all_sync(0xffffffffu, gm_wait(&sb->full[sa], pha, sb, a.status, 40 + (int)sa));
                if (!ok) break;
                ptx::tc_fence_after();
                const uint32_t sn = sa + 1 == NS ? 0u : sa + 1, phn = sa + 1 == NS ? pha ^ 1u : pha;
                if (leader) {
                    const uint64_t da = da0 + (uint64_t)(sa * (kATileBytes >> 4));
#pragma unroll
                    for (int p = 0; p < P; ++p) {  // int4: the hi tile, then the lo tile, against the same x stage
                        const uint64_t db = db0 + (uint64_t)((sa * P + p) * (kBTileBytes >> 4));
#pragma unroll
                        for (int k16 = 0; k16 < kBK / 16; ++k16)
                            ptx::umma_bf16(acc0, da + (uint64_t)(k16 * 2), db + (uint64_t)(k16 * 128), ti.halves == 2 ? idesc : idesc - less,
                                           accumulate | (uint32_t)(k16 + p));
                        if (ti.halves == 2) {
#pragma unroll
                            for (int k16 = 0; k16 < kBK / 16; ++k16)
                                ptx::umma_bf16(acc0 + kBN, da + (uint64_t)((kAHalfBytes >> 4) + k16 * 2),
                                               db + (uint64_t)(k16 * 128), idesc - less, accumulate | (uint32_t)(k16 + p));
                        }
                    }
                }
                ready = ptx::mbar_test_wait(ptx::smem_u32(&sb->full[sn]), phn);
                if (leader) ptx::umma_commit(ptx::smem_u32(&sb->empty[sa]));
                ready = __all_sync(0xffffffffu, ready);
                accumulate = 1;
                sa = sn;
                pha = phn;
            }
            if (!ok) break;
            if (leader) {
                if (use0) ptx::umma_commit(ptx::smem_u32(&sb->t_full[0]));
                if (use1) ptx::umma_commit(ptx::smem_u32(&sb->t_full[1]));
            }
            uses0 += use0;
            uses1 += use1;
        }
        // drain: every issued MMA must have completed before TMEM is released
        if (leader) {
            ptx::umma_commit(ptx::smem_u32(&sb->drain));
            (void)ptx::mbar_wait(ptx::smem_u32(&sb->drain), 0);
        }
        __syncwarp();
    } else if (warp >= kWarpEpi0 && warp < kWarpEpi0 + kEpiWarps) {
        // ------------------------------ epilogue ------------------------------
        const int quarter = warp & 3;                 // TMEM lanes 32*quarter .. +31 are the ones this warp may read
        const int grp = (warp - kWarpEpi0) >> 2;      // which accumulator this warp drains
        constexpr bool per_channel = (MODE == B200MOE_CT_INT8);
        const bool has_offset = per_channel && a.offset != nullptr;
        uint32_t use = 0, next1 = 0, seq = 0;
        for (;;) {
            TileInfo ti;
            if (!__all_sync(0xffffffffu, next_tile<RESOLVED>(sb, seq, ti, tile_prefix, row_start, a.G, n_nt, a.status))) break;
            // a two-half tile: this group takes row half `grp`; a one-half tile sits in one accumulator
            bool mine = true;
            int half = grp;
            if (ti.halves == 1) {
                mine = (int)next1 == grp;
                half = 0;
                next1 ^= 1u;
            }
            if (!mine) continue;
            // int8: every thread needs the scale (and scale * offset) of all 256 columns of the tile; the
            // warp stages them in its own shared-memory strip while the tile is still being accumulated
            float* es = epi_scale + (warp - kWarpEpi0) * kEpiScaleFloats;
            if (per_channel) {
                const size_t c0 = (size_t)ti.g * a.N + ti.n0;
#pragma unroll
                for (int i = 0; i < kBN / 32; ++i) {
                    const int col = i * 32 + lane;
                    const float sv = __bfloat162float(static_cast<const __nv_bfloat16*>(a.scale)[c0 + col]);
                    es[col] = sv;
                    es[kBN + col] = has_offset ? sv * __bfloat162float(a.offset[c0 + col]) : 0.f;
                }
                __syncwarp();
            }
            if constexpr (MODE == kCtInt4F16) {
                if (quarter == 0 && half == 0)  // one warp a tile, while it is being accumulated
                    int4_check_tile(a.row_exp, static_cast<const uint4*>(a.scale), a.K >> 7, a.N >> 3, ti.g, ti.row0, ti.rows, ti.n0, a.redo, a.redo_ctl);
            }
            if (!__all_sync(0xffffffffu, gm_wait(&sb->t_full[grp], use & 1, sb, a.status, 60 + grp))) break;
            ++use;
            ptx::tc_fence_after();
            {
                // (M = 64 leaves row i in TMEM lane 32 * (i / 16) + i % 16)
                const bool half_m = T::kShortRows > 0 && ti.rows - half * kBM <= T::kShortRows;
                int row;
                bool row_ok;
                if constexpr (T::kNibbles) {
                    // one number for both (0 .. 18 bytes of spills; with two, as below, 44 .. 80, and stored fp4 lost 5 to 10 % on short calls)
                    int at = half * kBM + quarter * 32 + lane;
                    if (half_m) at = half * kBM + ((lane & 16) << 4) + quarter * 16 + (lane & 15);  // (lanes from 16 on: past any tile's rows)
                    row = ti.row0 + at;
                    row_ok = at < ti.rows;
                } else {
                    row = ti.row0 + half * kBM + (half_m ? quarter * 16 + (lane & 15) : quarter * 32 + lane);
                    row_ok = row < ti.row0 + ti.rows && !(half_m && lane >= 16);
                }
                float unit = 1.f;  // (a row that is not exact in f16 comes out as zeros here)
                if constexpr (MODE == kCtInt4F16) unit = row_ok ? int4_row_unit(__ldca(a.row_exp + row)) : 0.f;
                const float rs = (has_offset && row_ok) ? __ldca(a.rowsum + row) : 0.f;
                if constexpr (SILU) {
                    __nv_bfloat16* arow = a.y + (size_t)row * (a.N >> 1) + (ti.n0 >> 1);
                    const uint32_t acc = tmem_base + grp * kBN + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
                    for (int c = 0; c < kBN / 32; ++c) {  // 16 activation columns per step
                        uint32_t rg[16], ru[16];
                        ptx::tmem_ld_32x16(acc + c * 16, rg);
                        ptx::tmem_ld_32x16(acc + kBN / 2 + c * 16, ru);
                        ptx::tmem_ld_wait();
                        uint32_t o[8];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t g01, g23, u01, u23;
                            if constexpr (per_channel) {
                                const float4 sg = *reinterpret_cast<const float4*>(es + c * 16 + 4 * q);
                                const float4 og = *reinterpret_cast<const float4*>(es + kBN + c * 16 + 4 * q);
                                const float4 su = *reinterpret_cast<const float4*>(es + kBN / 2 + c * 16 + 4 * q);
                                const float4 ou = *reinterpret_cast<const float4*>(es + kBN + kBN / 2 + c * 16 + 4 * q);
                                // accumulator positions (0,2,1,3) of a group of four hold columns 0..3
                                g01 = pack_bf16x2(fmaf(og.x, rs, sg.x * s8_sum(rg[4 * q])),
                                                  fmaf(og.y, rs, sg.y * s8_sum(rg[4 * q + 2])));
                                g23 = pack_bf16x2(fmaf(og.z, rs, sg.z * s8_sum(rg[4 * q + 1])),
                                                  fmaf(og.w, rs, sg.w * s8_sum(rg[4 * q + 3])));
                                u01 = pack_bf16x2(fmaf(ou.x, rs, su.x * s8_sum(ru[4 * q])),
                                                  fmaf(ou.y, rs, su.y * s8_sum(ru[4 * q + 2])));
                                u23 = pack_bf16x2(fmaf(ou.z, rs, su.z * s8_sum(ru[4 * q + 1])),
                                                  fmaf(ou.w, rs, su.w * s8_sum(ru[4 * q + 3])));
                            } else {
                                auto two = [&](const uint32_t (&r)[16], int c) {
                                    return pack_bf16x2(__uint_as_float(r[acc_pos<MODE>(c)]), __uint_as_float(r[acc_pos<MODE>(c + 1)]));
                                };
                                g01 = two(rg, 4 * q);
                                g23 = two(rg, 4 * q + 2);
                                u01 = two(ru, 4 * q);
                                u23 = two(ru, 4 * q + 2);
                            }
                            const uint32_t gw[2] = {g01, g23}, uw[2] = {u01, u23};
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const float g0 = __uint_as_float(gw[i] << 16), g1 = __uint_as_float(gw[i] & 0xFFFF0000u);
                                const float u0 = __uint_as_float(uw[i] << 16), u1 = __uint_as_float(uw[i] & 0xFFFF0000u);
                                o[2 * q + i] = pack_bf16x2(g0 / (1.f + __expf(-g0)) * u0, g1 / (1.f + __expf(-g1)) * u1);
                            }
                        }
                        if (row_ok) {
                            uint4* dst = reinterpret_cast<uint4*>(arow + c * 16);
                            dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
                            dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
                        }
                    }
                } else {
                __nv_bfloat16* yrow = a.y + (size_t)row * a.N + ti.n0;
#pragma unroll 1
                for (int c = 0; c < kBN / 32; ++c) {
                    if (MODE == B200MOE_CT_FP8 && ti.n0 + c * 32 >= a.N) break;  // 128-column last tile
                    uint32_t r[32];
                    ptx::tmem_ld_32x32(tmem_base + grp * kBN + c * 32 + ((uint32_t)(quarter * 32) << 16), r);
                    ptx::tmem_ld_wait();
                    uint32_t o[16];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {  // output columns 4q .. 4q+3 of the chunk
                        float4 s4 = make_float4(1.f, 1.f, 1.f, 1.f), o4 = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (per_channel) {
                            s4 = *reinterpret_cast<const float4*>(es + c * 32 + 4 * q);
                            o4 = *reinterpret_cast<const float4*>(es + kBN + c * 32 + 4 * q);
                        }
                        float v0 = __uint_as_float(r[acc_pos<MODE>(4 * q)]), v1 = __uint_as_float(r[acc_pos<MODE>(4 * q + 1)]);
                        float v2 = __uint_as_float(r[acc_pos<MODE>(4 * q + 2)]), v3 = __uint_as_float(r[acc_pos<MODE>(4 * q + 3)]);
                        if (per_channel) {
                            v0 = fmaf(o4.x, rs, s4.x * (kS8Unit * v0));
                            v1 = fmaf(o4.y, rs, s4.y * (kS8Unit * v1));
                            v2 = fmaf(o4.z, rs, s4.z * (kS8Unit * v2));
                            v3 = fmaf(o4.w, rs, s4.w * (kS8Unit * v3));
                        }
                        if constexpr (MODE == kCtInt4F16) { v0 *= unit; v1 *= unit; v2 *= unit; v3 *= unit; }
                        o[2 * q] = pack_bf16x2(v0, v1);
                        o[2 * q + 1] = pack_bf16x2(v2, v3);
                    }
                    if (row_ok) {
                        uint4* dst = reinterpret_cast<uint4*>(yrow + c * 32);
#pragma unroll
                        for (int q = 0; q < 4; ++q) dst[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                    }
                }
                }
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&sb->t_empty[grp]));
        }
    } else if (warp >= kWarpDq0 && !T::kDirect) {
        // ------------------------------ dequant ------------------------------
        // A unit of work is one stage (one k block); for int4 it holds the hi and the lo tile.  These
        // warps bound the kernel when tiles are small, so the loop carries as little bookkeeping as it
        // can: a stage counter, one iterator (for the loads, kPrefetch units ahead) whose global address
        // advances by a constant inside a tile, and shared addresses derived from one per-thread offset.
        const int dq_tid = threadIdx.x - kWarpDq0 * 32;
        const int grp = dq_tid / (kDqGroupWarps * 32);
        const DqLane d = dq_lane<MODE>(dq_tid % (kDqGroupWarps * 32));
        DqIter pf;
        pf.seq = 0;
        {
            TileInfo ti;
            pf.valid = next_tile<RESOLVED>(sb, pf.seq, ti, tile_prefix, row_start, a.G, n_nt, a.status);
            pf.g = ti.g;
            pf.n0 = ti.n0;
        }
        pf.kt = 0;
        dq_locate<MODE, SPLIT>(pf, weight, a, d);
        if (grp > 0 && pf.valid) dq_advance<MODE, SPLIT, RESOLVED>(pf, grp, weight, a, d, n_kt, tile_prefix, row_start, n_nt, sb);
        PackedRegs<MODE> regs[kPrefetch];
        bool loaded[kPrefetch];
#pragma unroll
        for (int u = 0; u < kPrefetch; ++u) {
            loaded[u] = pf.valid;
            if (pf.valid) {
                load_packed<MODE, SPLIT>(regs[u], pf, a, d);
                dq_advance<MODE, SPLIT, RESOLVED>(pf, kDqGroups, weight, a, d, n_kt, tile_prefix, row_start, n_nt, sb);
            }
        }
        const uint32_t sa0 = ptx::smem_u32(b_ring) + (T::kEightRows ? btile_offset(d.k0, d.chunk)
                                                                            : btile_offset(d.row, 2 * d.c16));
        uint32_t ib = grp;
        bool ok = true;
        while (ok) {
#pragma unroll
            for (int u = 0; u < kPrefetch; ++u) {
                if (!loaded[u]) { ok = false; break; }  // the schedule has ended
                const uint32_t slot = ib % NS;
                Int4Scales sc4;
                if constexpr (MODE == B200MOE_CT_INT4) sc4 = load_int4_scales(a, regs[u].e[0]);  // (late: registers)
                uint4 s8;
                if constexpr (MODE == kCtInt4F16) s8 = __ldg(static_cast<const uint4*>(a.scale) + regs[u].e[0]);
                bool got = true;
                if (ib >= NS) got = gm_wait(&sb->empty[slot], ((ib / NS) & 1) ^ 1, sb, a.status, 80 + (int)slot);
                if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
                const uint32_t sa = sa0 + slot * (uint32_t)(P * kBTileBytes);
                if constexpr (MODE == B200MOE_CT_INT4)
                    convert_block_int4(regs[u], sc4, sa, sa + kBTileBytes);
                else if constexpr (MODE == kCtInt4F16)
                    convert_int4_f16(regs[u], s8, sa);
                else if constexpr (MODE == kCtFp4Ascend)
                    convert_stage_fp4_ascend(regs[u], sa);
                else
                    convert_stage<MODE>(regs[u], sa);
                ptx::fence_proxy_async_smem();  // generic-proxy writes -> visible to the tensor core (async proxy)
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&sb->full[slot]));
                loaded[u] = pf.valid;
                if (pf.valid) {
                    load_packed<MODE, SPLIT>(regs[u], pf, a, d);
                    dq_advance<MODE, SPLIT, RESOLVED>(pf, kDqGroups, weight, a, d, n_kt, tile_prefix, row_start, n_nt, sb);
                }
                ib += kDqGroups;
            }
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == kWarpMma) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, kTmemCols);
    }
}

// Rows in use = end of the last group (clamped to M), by a whole CTA: a warp-level reduction, then one shared
// atomic per warp.
__device__ __forceinline__ int used_rows(const long long* __restrict__ group_list, int G, int gl_type, int M) {
    __shared__ int s_used;
    if (threadIdx.x == 0) s_used = 0;
    __syncthreads();
    long long v = 0;
    for (int g = threadIdx.x; g < G; g += blockDim.x) {
        const long long c = group_list[g];
        if (gl_type == B200MOE_GROUP_LIST_COUNTS) v += c > 0 ? c : 0; else v = c > v ? c : v;
    }
    v = v > M ? M : v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long other = __shfl_xor_sync(0xffffffffu, v, o);
        if (gl_type == B200MOE_GROUP_LIST_COUNTS) v += other; else v = other > v ? other : v;
    }
    v = v > M ? M : v;
    if ((threadIdx.x & 31) == 0 && v > 0) {
        if (gl_type == B200MOE_GROUP_LIST_COUNTS) atomicAdd(&s_used, (int)v); else atomicMax(&s_used, (int)v);
    }
    __syncthreads();
    return (s_used < 0 || s_used > M) ? M : s_used;  // (a sum of eight clamped parts could wrap)
}

// Row sums of x in fp32 (the offset term of the int8 epilogue): one warp per row.  Rows past the
// last group are skipped (a caller may pass a buffer sized for the worst case as x).  Being the first kernel of its
// call, it also zeroes status words 0 .. 3, which saves the call a memset of its own, and lets the GEMM start its
// prologue beside it (4 experts, 128 rows, 256 x 512: 18.1 -> 12.3 us).
__global__ void rowsum_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ out, int M, int K,
                              const long long* __restrict__ group_list, int G, int gl_type, int* __restrict__ status) {
    grid_dep_launch();
    if (blockIdx.x == 0 && threadIdx.x < 4) status[threadIdx.x] = 0;
    const int used = used_rows(group_list, G, gl_type, M);
    const int wpb = blockDim.x >> 5;
    for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < used; row += gridDim.x * wpb) {
        const uint4* p = reinterpret_cast<const uint4*>(x + (size_t)row * K);
        float s = 0.f;
        for (int i = threadIdx.x & 31; i < K / 8; i += 32) {
            const uint4 q = __ldg(p + i);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) s += __uint_as_float(w[j] << 16) + __uint_as_float(w[j] & 0xFFFF0000u);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) out[row] = s;
    }
}

// Grid of the row-sum kernel: one warp per row up to a few CTAs per multiprocessor, then a stride
// (every CTA first reduces the group list, which should not be repeated thousands of times).
static unsigned rowsum_blocks(int64_t M) {
    const int64_t want = (M + 7) / 8, cap = 16LL * sm_count();
    return (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
}

void launch_rowsum(const void* x, float* out, int64_t M, int64_t K, const int64_t* group_list, int64_t G, int gl_type,
                   int* status, cudaStream_t stream) {
    rowsum_kernel<<<rowsum_blocks(M), 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), out, (int)M, (int)K,
                                                        reinterpret_cast<const long long*>(group_list), (int)G, gl_type, status);
}

// One-pass int4: a row of x as f16 times 2^-e, e into row_exp (kRowNotF16: not exact).
// One warp a row; the row's second reading comes from L1 or L2, so the bound is its bytes in and out.
__global__ void __launch_bounds__(256)
gm_int4_prepare_x_kernel(const __nv_bfloat16* __restrict__ x, uint16_t* __restrict__ x16, int* __restrict__ row_exp, int M, int K,
                         const long long* __restrict__ group_list, int G, int gl_type, int* __restrict__ status,
                         int* __restrict__ ctl) {
    grid_dep_launch();
    if (blockIdx.x == 0 && threadIdx.x < 4) status[threadIdx.x] = 0;
    const int used = used_rows(group_list, G, gl_type, M);
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5, n_vec = K / 8;
    for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < used; row += gridDim.x * wpb) {
        const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)row * K);
        uint4* dst = reinterpret_cast<uint4*>(x16 + (size_t)row * K);
        uint32_t mx = 0u;  // bf16 magnitudes order like integers
#pragma unroll 8
        for (int i = lane; i < n_vec; i += 32) {
            const uint4 q = __ldg(src + i);
            mx = __vmaxu2(__vmaxu2(mx, __vmaxu2(q.x & 0x7FFF7FFFu, q.y & 0x7FFF7FFFu)), __vmaxu2(q.z & 0x7FFF7FFFu, q.w & 0x7FFF7FFFu));
        }
        mx = __reduce_max_sync(0xffffffffu, max(mx & 0xFFFFu, mx >> 16));
        const int e_max = (int)(mx >> 7);  // biased exponent of the largest magnitude
        const int e = mx == 0u ? 0 : e_max - 127 - 14;
        // (2^-e and the epilogue's 2^(e - 6) are normal numbers)
        bool ok = mx == 0u || (e_max >= 32 && e_max < 255);
        const float down = ok ? __uint_as_float((uint32_t)(127 - e) << 23) : 0.f;
#pragma unroll 4
        for (int i = lane; i < n_vec; i += 32) {
            const uint4 q = __ldg(src + i);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
            uint32_t h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float f0 = __uint_as_float(w[j] << 16) * down, f1 = __uint_as_float(w[j] & 0xFFFF0000u) * down;
                const __half2 hh = __floats2half2_rn(f0, f1);
                h[j] = *reinterpret_cast<const uint32_t*>(&hh);
                // exact: the same value back, and no zero that was none (f0, f1 themselves may underflow)
                const float2 back = __half22float2(hh);
                ok = ok && back.x == f0 && back.y == f1 && ((h[j] & 0x7FFFu) != 0u) == ((w[j] & 0x7FFFu) != 0u) &&
                     ((h[j] & 0x7FFF0000u) != 0u) == ((w[j] & 0x7FFF0000u) != 0u);
            }
            dst[i] = make_uint4(h[0], h[1], h[2], h[3]);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) {
            row_exp[row] = ok ? e : kRowNotF16;
            if (!ok) atomicAdd(ctl + 2, 1);
        }
    }
}

// int8 tiles of fewer than 32 stages are resolved by the publisher.  Each role | publisher, us: 4 experts of 32 rows, 256 x 512: 13.2 |
// 12.3; 32 of 300, 64 x 2048: 45.0 | 41.0; 128 experts, 32768 rows by popularity, 1024 x 4096: 489 | 474, its SiLU form 526 | 513; 64 of
// 210, 1536 x 2048: 139.2 | 137.4, SiLU 154.7 | 155.9, 2048 x 2048: 172.6 | 170.8, SiLU 189.9 | 191.2; 128 of 32, 4096 x 2048: 363 |
// 378, SiLU 376 | 398.
constexpr int kInt8RolesK = 2048;

// Whether a call of int4 without offsets goes through f16 in one pass: where the tiles of a multiprocessor come to at least 48 stages of 64 k, the
// preparation of x and the two launches more (6 .. 10 us, and the bytes of x twice) are won back; where whole experts are long and N is a
// single column tile, they are not, nor where short ones make a single wave, which waits for its stages'
// round trips and not for MMAs.  us, hi and lo | one pass, back to back, experts : rows : K x N (even lists unless said): 128 : 8192 : 2048 x 256 50.9 |
// 69.8; 32 : 1056 : 4096 x 1024 87.0 | 102.3; 16 : 528 : 7168 x 2048 142.1 | 167.6; 20 : 800 : 4096 x 2048 158.8 | 92.0; 8 : 1024 : 2048 x 2048
// (32 stages) 49.5 | 59.7; 32 : 1024 : 2048 x 1024 (32) 47.5 | 56.5; 16 : 4096 : 256 x 4096 (16) 45.4 | 44.4; 16 : 1024 : 256 x 1024 (4) 16.6 | 23.1;
// 64 : 4096 by popularity : 1024 x 1024 (48) 64.3 | 52.8; 32 : 256 : 7168 x 2048 (224) 264 | 184; 256 : 1024 : 2048 x 2048 (448) 554 | 345; 64 : 8192 by
// popularity : 7168 x 1024 409.6 | 330.9; 256 : 8192 : 2048 x 7168 1992 | 1226; 256 : 65536 by popularity : 7168 x 4096 8840 | 5586.
static bool int4_one_pass(int64_t M, int64_t K, int64_t N, int64_t G) {
    const int64_t tiles = N / kBN * (M / kTileM + (M < G ? M : G)), sms = sm_count();  // (all experts have rows)
    const bool long_experts = M > 64 * G;
    return (tiles + sms - 1) / sms * (K / kBK) >= 48 && (long_experts ? N >= 2 * kBN : N / kBN * (M < G ? M : G) > sms);
}

static size_t gm_smem_bytes(int G) {
    return 1024 + (size_t)kNS * (kATileBytes + kBTileBytes) + kBarrierBytes + sizeof(float) * kEpiWarps * kEpiScaleFloats +
           sizeof(int) * 3 * (size_t)(G + 1);
}

template <int MODE, bool SILU = false, bool RESOLVED = GmTraits<MODE>::kResolved>
static int gm_launch(const void* x, const void* w, const GemmArgs& a, cudaStream_t stream) {
    using T = GmTraits<MODE>;
    if (MODE == B200MOE_CT_INT8 && !RESOLVED && a.K < kInt8RolesK) return gm_launch<MODE, SILU, true>(x, w, a, stream);
    CUtensorMap tx, txs, tw;
    int rc = make_tensor_map_2d(&tx, x, 2, (uint64_t)a.M, a.K, kBM, kBK, true);
    if (rc != B200MOE_OK) return rc;
    rc = make_tensor_map_2d(&txs, x, 2, (uint64_t)a.M, a.K, kSmallRows, kBK, true);
    if (rc != B200MOE_OK) return rc;
    if (T::kDirect)
        rc = make_tensor_map_2d(&tw, w, 2, (uint64_t)a.G * a.K, a.N, kBK, 64, true);
    else
        rc = make_tensor_map_2d(&tw, w, 1, (uint64_t)a.G * a.K, T::kNibbles ? a.N / 2 : a.N, kBK,
                                SILU && MODE == kCtFp4E8m0 ? kBN / 4  // gate and up halves of a tile: two boxes
                                : a.N < kBN ? (uint32_t)(T::kNibbles ? a.N / 2 : a.N) : (uint32_t)T::kPRowBytes, false);
    if (rc != B200MOE_OK) return rc;
    const size_t smem = gm_smem_bytes(a.G);
    B200MOE_CUDA_TRY(cudaFuncSetAttribute(grouped_gemm_kernel<MODE, SILU, RESOLVED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
    if (a.rowsum != nullptr || a.redo_ctl != nullptr) {  // the kernel before is launch_rowsum's, or one of one-pass int4
        B200MOE_CUDA_TRY(launch_dependent(grouped_gemm_kernel<MODE, SILU, RESOLVED>, (unsigned)sm_count(), kGemmThreads, smem, stream, tx, txs, tw,
                                          static_cast<const uint8_t*>(w), a));
    } else {
        grouped_gemm_kernel<MODE, SILU, RESOLVED><<<sm_count(), kGemmThreads, smem, stream>>>(tx, txs, tw, static_cast<const uint8_t*>(w), a);
        B200MOE_CUDA_TRY(cudaGetLastError());
    }
    return B200MOE_OK;
}

static size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

// Scratch of a one-pass int4 call: control words, row exponents, the list of tiles to do again, x as f16.
struct Int4Scratch {
    size_t exp, redo, x16, bytes;
};
static Int4Scratch int4_scratch(int64_t M, int64_t K, int64_t N, int64_t G) {
    const size_t tiles = (size_t)(N / kBN) * (size_t)(M / kTileM + (M < G ? M : G));  // at most
    Int4Scratch s;
    s.exp = 256;
    s.redo = s.exp + align256((size_t)M * sizeof(int));
    s.x16 = s.redo + align256(tiles * sizeof(int4));
    s.bytes = s.x16 + (size_t)M * (size_t)K * 2;
    return s;
}

}  // namespace b200moe

using namespace b200moe;

extern "C" size_t b200moe_grouped_gemm_workspace_bytes(int64_t M, int64_t K, int64_t N, int64_t G, int compute_type,
                                                       int weight_layout) {
    size_t b = B200MOE_STATUS_BYTES;
    if (compute_type == B200MOE_CT_INT8) b += align256((size_t)M * sizeof(float));
    (void)K; (void)N; (void)G; (void)weight_layout;  // stored-order fp4 weights are read in place
    return b;
}

extern "C" size_t b200moe_grouped_gemm_scratch_bytes(int64_t M, int64_t K, int64_t N, int64_t G, int compute_type, int has_offset) {
    if (compute_type != B200MOE_CT_INT4 || M <= 0 || K <= 0 || N <= 0 || G <= 0 || (K % 128) != 0 || (N % kBN) != 0) return 0;
    if (has_offset != 0 || !int4_one_pass(M, K, N, G)) return 0;
    return int4_scratch(M, K, N, G).bytes;
}

extern "C" int b200moe_grouped_gemm(const void* x, const void* weight, const void* scale, const void* offset,
                                    const int64_t* group_list, void* y, int64_t M, int64_t K, int64_t N, int64_t G,
                                    int compute_type, int group_list_type, int weight_layout, void* workspace,
                                    size_t workspace_bytes, void* stream) {
    return b200moe_grouped_gemm_scratch(x, weight, scale, offset, group_list, y, M, K, N, G, compute_type, group_list_type,
                                        weight_layout, workspace, workspace_bytes, nullptr, 0, stream);
}

extern "C" int b200moe_grouped_gemm_scratch(const void* x, const void* weight, const void* scale, const void* offset,
                                            const int64_t* group_list, void* y, int64_t M, int64_t K, int64_t N, int64_t G,
                                            int compute_type, int group_list_type, int weight_layout, void* workspace,
                                            size_t workspace_bytes, void* scratch, size_t scratch_bytes, void* stream) {
    if (compute_type < B200MOE_CT_FP8 || compute_type > B200MOE_CT_BF16) return B200MOE_ERR_COMPUTE_TYPE;
    if (group_list_type != B200MOE_GROUP_LIST_CUMSUM && group_list_type != B200MOE_GROUP_LIST_COUNTS)
        return B200MOE_ERR_ARGUMENT;
    if (weight_layout != B200MOE_LAYOUT_CANONICAL && weight_layout != B200MOE_LAYOUT_ASCEND)
        return B200MOE_ERR_ARGUMENT;
    if (M < 0 || K <= 0 || N <= 0 || G <= 0 || G > kMaxExperts || M > 0x7FFFFFF0LL || K > 0x7FFFFFF0LL ||
        N > 0x7FFFFFF0LL || G * K > 0x7FFFFFF0LL)
        return B200MOE_ERR_SHAPE;
    // fp8: what the reference takes (K and N multiples of its 128 x 128 scale block: a last tile of
    // 128 columns); the other modes work on whole 256-column tiles
    if (compute_type == B200MOE_CT_FP8 ? ((K % 128) != 0 || (N % 128) != 0) : ((K % kBK) != 0 || (N % kBN) != 0))
        return B200MOE_ERR_SHAPE;
    if (compute_type == B200MOE_CT_INT4 && (K % 128) != 0) return B200MOE_ERR_SHAPE;
    if (M == 0) return B200MOE_OK;
    const bool needs_scale = compute_type != B200MOE_CT_BF16;
    if (!x || !weight || (needs_scale && !scale) || !group_list || !y) return B200MOE_ERR_NULL_POINTER;
    if (!aligned16(x) || !aligned16(weight) || (scale && !aligned16(scale)) || !aligned16(y) || (offset && !aligned16(offset)))
        return B200MOE_ERR_ALIGNMENT;
    const size_t need = b200moe_grouped_gemm_workspace_bytes(M, K, N, G, compute_type, weight_layout);
    if (workspace == nullptr || workspace_bytes < need || !aligned16(workspace)) return B200MOE_ERR_WORKSPACE;

    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t scratch_need = b200moe_grouped_gemm_scratch_bytes(M, K, N, G, compute_type, offset != nullptr);
    const bool one_pass = scratch_need != 0 && scratch != nullptr && scratch_bytes >= scratch_need && aligned16(scratch);
    // (the row sums' kernel zeroes the status words itself, and so does the one that prepares x for one-pass int4)
    if (one_pass) B200MOE_CUDA_TRY(cudaMemsetAsync(scratch, 0, 16, s));
    else if (compute_type != B200MOE_CT_INT8 || offset == nullptr) B200MOE_CUDA_TRY(cudaMemsetAsync(workspace, 0, 16, s));
    uint8_t* ws = static_cast<uint8_t*>(workspace) + B200MOE_STATUS_BYTES;
    GemmArgs a;
    a.scale = scale;
    a.offset = nullptr;
    a.rowsum = nullptr;
    a.group_list = group_list;
    a.y = static_cast<__nv_bfloat16*>(y);
    a.M = (int)M; a.K = (int)K; a.N = (int)N; a.G = (int)G;
    a.gl_type = group_list_type;
    a.status = static_cast<int*>(workspace);

    if (compute_type == B200MOE_CT_INT8) {
        float* rowsum = reinterpret_cast<float*>(ws);
        ws += align256((size_t)M * sizeof(float));
        if (offset != nullptr) {
            launch_rowsum(x, rowsum, M, K, group_list, G, group_list_type, a.status, s);
            B200MOE_CUDA_TRY(cudaGetLastError());
            a.offset = static_cast<const __nv_bfloat16*>(offset);
            a.rowsum = rowsum;
        }
        return gm_launch<B200MOE_CT_INT8>(x, weight, a, s);
    }
    if (compute_type == B200MOE_CT_INT4) {
        a.offset = static_cast<const __nv_bfloat16*>(offset);  // folded into the weights by the dequant warps
        if (!one_pass) return gm_launch<B200MOE_CT_INT4>(x, weight, a, s);
        const Int4Scratch at = int4_scratch(M, K, N, G);
        uint8_t* sc = static_cast<uint8_t*>(scratch);
        int* exps = reinterpret_cast<int*>(sc + at.exp);
        void* x16 = sc + at.x16;
        a.row_exp = exps;
        a.redo = reinterpret_cast<int4*>(sc + at.redo);
        a.redo_ctl = reinterpret_cast<int*>(sc);
        gm_int4_prepare_x_kernel<<<rowsum_blocks(M), 256, 0, s>>>(
            static_cast<const __nv_bfloat16*>(x), static_cast<uint16_t*>(x16), exps, (int)M, (int)K,
            reinterpret_cast<const long long*>(group_list), (int)G, group_list_type, a.status, a.redo_ctl);
        B200MOE_CUDA_TRY(cudaGetLastError());
        const int rc = gm_launch<kCtInt4F16>(x16, weight, a, s);
        return rc != B200MOE_OK ? rc : gm_launch<B200MOE_CT_INT4>(x, weight, a, s);
    }
    if (compute_type == B200MOE_CT_FP8) return gm_launch<B200MOE_CT_FP8>(x, weight, a, s);
    if (compute_type == B200MOE_CT_BF16) return gm_launch<B200MOE_CT_BF16>(x, weight, a, s);
    // the stored ("ascend") order is read in place by the dequant warps
    if (weight_layout == B200MOE_LAYOUT_ASCEND) return gm_launch<kCtFp4Ascend>(x, weight, a, s);
    return gm_launch<B200MOE_CT_FP4>(x, weight, a, s);
}

extern "C" int b200moe_grouped_gemm_int8_silu(const void* x, const void* weight, const void* scale, const void* offset,
                                              const int64_t* group_list, void* out, int64_t M, int64_t K, int64_t N,
                                              int64_t G, int group_list_type, void* workspace, size_t workspace_bytes,
                                              void* stream) {
    if (group_list_type != B200MOE_GROUP_LIST_CUMSUM && group_list_type != B200MOE_GROUP_LIST_COUNTS)
        return B200MOE_ERR_ARGUMENT;
    if (M < 0 || K <= 0 || N <= 0 || G <= 0 || G > kMaxExperts || M > 0x7FFFFFF0LL || K > 0x7FFFFFF0LL ||
        N > 0x7FFFFFF0LL || G * K > 0x7FFFFFF0LL)
        return B200MOE_ERR_SHAPE;
    if ((K % kBK) != 0 || (N % kBN) != 0) return B200MOE_ERR_SHAPE;
    if (M == 0) return B200MOE_OK;
    if (!x || !weight || !scale || !group_list || !out) return B200MOE_ERR_NULL_POINTER;
    if (!aligned16(x) || !aligned16(weight) || !aligned16(scale) || !aligned16(out) || (offset && !aligned16(offset)))
        return B200MOE_ERR_ALIGNMENT;
    const size_t need = b200moe_grouped_gemm_workspace_bytes(M, K, N, G, B200MOE_CT_INT8, B200MOE_LAYOUT_CANONICAL);
    if (workspace == nullptr || workspace_bytes < need || !aligned16(workspace)) return B200MOE_ERR_WORKSPACE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (offset == nullptr) B200MOE_CUDA_TRY(cudaMemsetAsync(workspace, 0, 16, s));  // (else: launch_rowsum)
    GemmArgs a;
    a.scale = scale;
    a.offset = nullptr;
    a.rowsum = nullptr;
    a.group_list = group_list;
    a.y = static_cast<__nv_bfloat16*>(out);
    a.M = (int)M; a.K = (int)K; a.N = (int)N; a.G = (int)G;
    a.gl_type = group_list_type;
    a.status = static_cast<int*>(workspace);
    if (offset != nullptr) {
        float* rowsum = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + B200MOE_STATUS_BYTES);
        launch_rowsum(x, rowsum, M, K, group_list, G, group_list_type, a.status, s);
        B200MOE_CUDA_TRY(cudaGetLastError());
        a.offset = static_cast<const __nv_bfloat16*>(offset);
        a.rowsum = rowsum;
    }
    return gm_launch<B200MOE_CT_INT8, true>(x, weight, a, s);
}

extern "C" int b200moe_grouped_gemm_fp4_e8m0(const void* x, const void* codes, const void* scale_e8m0,
                                             const int64_t* group_list, void* out, int64_t M, int64_t K, int64_t N, int64_t G,
                                             int group_list_type, int gate_up_silu, void* workspace, size_t workspace_bytes,
                                             void* stream) {
    if (group_list_type != B200MOE_GROUP_LIST_CUMSUM && group_list_type != B200MOE_GROUP_LIST_COUNTS)
        return B200MOE_ERR_ARGUMENT;
    if (M < 0 || K <= 0 || N <= 0 || G <= 0 || G > kMaxExperts || M > 0x7FFFFFF0LL || K > 0x7FFFFFF0LL ||
        N > 0x7FFFFFF0LL || G * K > 0x7FFFFFF0LL)
        return B200MOE_ERR_SHAPE;
    if ((K % kBK) != 0 || (N % kBN) != 0) return B200MOE_ERR_SHAPE;
    if (M == 0) return B200MOE_OK;
    if (!x || !codes || !scale_e8m0 || !group_list || !out) return B200MOE_ERR_NULL_POINTER;
    if (!aligned16(x) || !aligned16(codes) || !aligned16(out)) return B200MOE_ERR_ALIGNMENT;
    const size_t need = b200moe_grouped_gemm_workspace_bytes(M, K, N, G, B200MOE_CT_FP4, B200MOE_LAYOUT_CANONICAL);
    if (workspace == nullptr || workspace_bytes < need || !aligned16(workspace)) return B200MOE_ERR_WORKSPACE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    B200MOE_CUDA_TRY(cudaMemsetAsync(workspace, 0, 16, s));
    GemmArgs a;
    a.scale = scale_e8m0;
    a.offset = nullptr;
    a.rowsum = nullptr;
    a.group_list = group_list;
    a.y = static_cast<__nv_bfloat16*>(out);
    a.M = (int)M; a.K = (int)K; a.N = (int)N; a.G = (int)G;
    a.gl_type = group_list_type;
    a.status = static_cast<int*>(workspace);
    return gate_up_silu ? gm_launch<kCtFp4E8m0, true>(x, codes, a, s) : gm_launch<kCtFp4E8m0>(x, codes, a, s);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant for callers that cannot allocate device memory
// ---------------------------------------------------------------------------------------------
// Some hosts of these kernels may not call cudaMalloc at all: a plug-in that runs inside another
// framework's execution step, where every device allocation is owned by that framework's arena and
// a foreign cudaMalloc would fragment or deadlock it; a real-time serving loop that forbids
// allocation after start-up.  The regular
// entry point asks such callers for a workspace they have no way to provide.  This one keeps the
// kernel's scratch (two status words and one fp32 row sum per row of x) in a fixed array that is
// part of the loaded library image, so the caller passes inputs and outputs only.
namespace b200moe {

constexpr long long kNoAllocMaxRows = 65536;
static __device__ __align__(256) unsigned char g_noalloc_scratch[B200MOE_STATUS_BYTES + kNoAllocMaxRows * sizeof(float)];

// Device address of the scratch array on the current device, resolved once per device.  The array's
// name is only a host-side handle: a kernel must be given the address cudaGetSymbolAddress returns.
// This lookup and the first launch of the kernel on a device (the driver loads the kernel image, with
// the array in it, at that point) are the set-up a warm-up call gets out of the way: callers make one
// call per device before their allocation-free phase and before any stream capture.  The cached
// address is valid for the life of the process, not across a device reset.
static int noalloc_scratch(void** out) {
    static void* addr[64];
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return B200MOE_ERR_CUDA;
    std::lock_guard<std::mutex> lock(mu);
    if (addr[dev] == nullptr) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || p == nullptr) {
            (void)cudaGetLastError();
            return B200MOE_ERR_CUDA;
        }
        addr[dev] = p;
    }
    *out = addr[dev];
    return B200MOE_OK;
}

}  // namespace b200moe

extern "C" int64_t b200moe_grouped_gemm_int8_noalloc_max_rows(void) { return kNoAllocMaxRows; }

extern "C" int b200moe_grouped_gemm_int8_noalloc(const void* x, const void* weight, const void* scale,
                                                 const void* offset, const int64_t* group_list, void* y, int64_t M,
                                                 int64_t K, int64_t N, int64_t G, int group_list_type, void* stream) {
    if (group_list_type != B200MOE_GROUP_LIST_CUMSUM && group_list_type != B200MOE_GROUP_LIST_COUNTS)
        return B200MOE_ERR_ARGUMENT;
    if (M < 0 || K <= 0 || N <= 0 || G <= 0 || G > kMaxExperts || K > 0x7FFFFFF0LL || N > 0x7FFFFFF0LL ||
        G * K > 0x7FFFFFF0LL)
        return B200MOE_ERR_SHAPE;
    if (M > kNoAllocMaxRows) return B200MOE_ERR_NOALLOC_LIMIT;
    if ((K % kBK) != 0 || (N % kBN) != 0) return B200MOE_ERR_SHAPE;
    if (M == 0) return B200MOE_OK;
    if (!x || !weight || !scale || !group_list || !y) return B200MOE_ERR_NULL_POINTER;
    if (!aligned16(x) || !aligned16(weight) || !aligned16(scale) || !aligned16(y) || (offset && !aligned16(offset)))
        return B200MOE_ERR_ALIGNMENT;

    void* scratch = nullptr;
    const int rc = noalloc_scratch(&scratch);
    if (rc != B200MOE_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // the array keeps whatever the previous call left: the status words must start at zero
    if (offset == nullptr) B200MOE_CUDA_TRY(cudaMemsetAsync(scratch, 0, 16, s));  // (else: launch_rowsum)
    GemmArgs a;
    a.scale = scale;
    a.offset = nullptr;
    a.rowsum = nullptr;
    a.group_list = group_list;
    a.y = static_cast<__nv_bfloat16*>(y);
    a.M = (int)M; a.K = (int)K; a.N = (int)N; a.G = (int)G;
    a.gl_type = group_list_type;
    a.status = static_cast<int*>(scratch);
    if (offset != nullptr) {
        float* rowsum = reinterpret_cast<float*>(static_cast<unsigned char*>(scratch) + B200MOE_STATUS_BYTES);
        launch_rowsum(x, rowsum, M, K, group_list, G, group_list_type, a.status, s);
        B200MOE_CUDA_TRY(cudaGetLastError());
        a.offset = static_cast<const __nv_bfloat16*>(offset);
        a.rowsum = rowsum;
    }
    return gm_launch<B200MOE_CT_INT8>(x, weight, a, s);
}

extern "C" int b200moe_noalloc_read_status(int32_t out[2], void* stream) {
    if (out == nullptr) return B200MOE_ERR_NULL_POINTER;
    void* scratch = nullptr;
    const int rc = noalloc_scratch(&scratch);
    if (rc != B200MOE_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    B200MOE_CUDA_TRY(cudaMemcpyAsync(out, scratch, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    B200MOE_CUDA_TRY(cudaStreamSynchronize(s));
    return B200MOE_OK;
}
