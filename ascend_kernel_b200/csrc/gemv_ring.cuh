// Grouped GEMV on the tensor core with its operands streamed through a shared-memory ring (part of grouped_gemv.cu).
//
// Two CTAs a multiprocessor, each a producer warp and 8 consumer warps.  The producer's lane draws the units (up to 8 rows of an
// expert, slab of 256 columns, part of the k range), and copies their stages by TMA: 64 k rows of the slab's
// packed weights, of the group scales (fp4) and of the unit's x rows.  It runs ahead of the consumers by the ring, over the
// end of a unit, so the next unit's first weights arrive while the sums of this one are being put together; with loads
// into registers a unit started cold: ticket, look-up, staging of x, first loads, each waited for in turn.
// Every consumer warp takes 16 k rows x 128 columns of each stage, or 32 x 64: eight mma.sync m16n8k16 with the weights as the 16 x 16
// operand and up to eight x rows as the other (a legacy instruction on purpose: the tile is 16 x 8 and HBM is the bound).
// us, register kernel | one CTA of 16 consumer warps and stages of 128 k | this, called in turn with the register kernel: int8, 32 tokens x 8
// over 256 experts, 7168 x 4096: 886 | 830, 875 | 784 (6.1 TB/s); stored fp4, 37 tokens x 8, 2048 x 7168: 427 | 376, 419 | 354 (4.6
// TB/s); fp8, one token on 8 experts, 7168 x 4096: 70.3 | 74.4, 70.2 | 63.5, 32 tokens x 8: 906 | 890 (5.4 TB/s; 968 with 16 x 128 a
// warp and the block's scale read in front of each stage).  One CTA leaves its multiprocessor without work
// while its sums are put together (1200 .. 1700 cycles a unit); what is left at two is issue slots (about 3 per fp8 weight, 2 per fp4
// and int8 one).
#pragma once

#include "ptx.cuh"

namespace b200moe {

constexpr int kRgK = 64;                          // k rows of a stage
constexpr int kRgWarps = 8;                       // consumers
constexpr int kRgThreads = (kRgWarps + 1) * 32;
constexpr int kRgRows = 8;                        // x rows per unit: the instruction's n
constexpr int kRgRun = 8;                         // int8: stages in one partial sum
constexpr int kRgXBytes = kRgRows * kRgK * 2;     // a swizzled box of 8 rows x 64 k
static_assert(kRgWarps * 32 == kGvSlabN, "one thread a column");
// A part's slot holds four rows' sums, or eight where an expert has more than four rows: then there is room for half as many parts, and
// there are half as many units as with passes of four rows.
constexpr int kRgSlotFloats = 2 * kGvSlotFloats;
static_assert(kRgSlotFloats >= kRgRows * (kGvSlabN + 1) && kGvSlotFloats >= kGvRows * (kGvSlabN + 1), "slot: sums of the columns, sums of x");

template <int MODE>
struct RgTraits {
    static constexpr bool kFp4 = MODE == B200MOE_CT_FP4;
    static constexpr int kWBytes = kRgK * (kFp4 ? kGvSlabN / 2 : kGvSlabN);
    static constexpr int kSBytes = kFp4 ? kRgK / 16 * kGvSlabN * 2 : 0;
    static constexpr int kStageBytes = kWBytes + kSBytes + kRgXBytes;
    static constexpr int kStages = kFp4 ? 7 : 5;
    // A warp's share of a stage: 16 k rows (one scale group) x 128 columns of fp4, 32 x 64 of the byte formats: the same
    // weights a lane, but the fp32 scaling of fp8 comes once for two chained instructions instead of for each, and the sums of two k groups
    // meet instead of four.
    static constexpr int kKGroups = kFp4 ? 4 : 2, kKRows = kRgK / kKGroups;  // warps along k, rows of each
    static constexpr int kCols = kGvSlabN * kKGroups / kRgWarps;             // columns of a warp
    static constexpr int kAcc = kCols / 16;                                  // 16 x 8 accumulators of a warp
    static constexpr int kRedRows = 16 / kKGroups;                           // rows whose sums are put together at a time
    static_assert(kWBytes % 1024 == 0 && kSBytes % 1024 == 0 && kRgXBytes % 1024 == 0, "swizzled boxes");
};

struct RgUnit {
    int g, r0, rows, n0;  // expert, first row, rows (0: no more units), first column
    int k0, k1;           // its part of the k range
    int n_split, split, slot;
    int pad;
};

struct RgBarriers {
    uint64_t full[8], empty[8];
    uint64_t unit_full[2], unit_empty[2];
    uint64_t sync;
    RgUnit unit[2];
    int abort, last;
    int per_pass, units, parts, part_rows, slot_rows;
    float xsum[4][kRgRows];
};

__device__ __noinline__ bool rg_wait_slow(uint32_t bar, uint32_t parity, RgBarriers* sb, int* status, int id) {
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
__device__ __forceinline__ bool rg_wait(uint64_t* bar, uint32_t parity, RgBarriers* sb, int* status, int id) {
    const uint32_t b = ptx::smem_u32(bar);
    if (ptx::mbar_try_wait(b, parity)) return true;
    return rg_wait_slow(b, parity, sb, status, id);
}
// The consumer warps among themselves.  (Not a hardware barrier: every wait here is bounded.)
__device__ __forceinline__ bool rg_sync(RgBarriers* sb, uint32_t& phase, int* status) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) ptx::mbar_arrive(ptx::smem_u32(&sb->sync));
    const bool ok = __all_sync(0xffffffffu, rg_wait(&sb->sync, phase, sb, status, 74));
    phase ^= 1u;
    return ok;
}

__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// Lane (g, t) = (lane / 4, lane % 4) holds, of every 16 k rows, {2t, 2t + 1, 2t + 8, 2t + 9} (the instruction's own k indices)
// of its columns, and of x row g; c[j]: columns 2j, 2j + 1 of the lane's x two x rows.
// Byte formats: a warp's 32 k rows x 64 columns of a stage; `w0`, `w1`: shared addresses of the lane's eight columns in rows 2t, 2t + 1
// (rows 8 apart are 1024 bytes apart and share their swizzle), b[h]: x of rows 16h ...
template <int MODE>
__device__ __forceinline__ void rg_step_bytes(uint32_t w0, uint32_t w1, const uint32_t (&b)[2][2], float sf, float (&c)[4][4]) {
    float d[4][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint2 q0 = lds64(w0 + h * 2048), q1 = lds64(w1 + h * 2048), q2 = lds64(w0 + h * 2048 + 1024), q3 = lds64(w1 + h * 2048 + 1024);
        const uint32_t r0w[2] = {q0.x, q0.y}, r1w[2] = {q1.x, q1.y}, r2w[2] = {q2.x, q2.y}, r3w[2] = {q3.x, q3.y};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
            for (int o = 0; o < 2; ++o) {  // byte pairs (0,1) and (2,3) of word i: accumulator j = 2i + o
                uint32_t a0, a1, a2, a3;
                if constexpr (MODE == B200MOE_CT_INT8) {
                    const uint32_t sel = o == 0 ? 0x5410u : 0x7632u;
                    s8x4_to_bf16_even_odd(prmt(r0w[i], r1w[i], sel), a0, a1);  // rows (2t, 2t+1) at the two columns
                    s8x4_to_bf16_even_odd(prmt(r2w[i], r3w[i], sel), a2, a3);  // rows (2t+8, 2t+9)
                } else {
                    // byte b of both rows into the high bytes of the two lanes (the low bytes are masked off)
                    const uint32_t s0 = o == 0 ? 0x4000u : 0x6020u, s1 = o == 0 ? 0x5010u : 0x7030u;
                    a0 = e4m3x2_hi_to_bf16(prmt(r0w[i], r1w[i], s0));
                    a1 = e4m3x2_hi_to_bf16(prmt(r0w[i], r1w[i], s1));
                    a2 = e4m3x2_hi_to_bf16(prmt(r2w[i], r3w[i], s0));
                    a3 = e4m3x2_hi_to_bf16(prmt(r2w[i], r3w[i], s1));
                }
                float (&dd)[4] = d[2 * i + o];
                if (h == 0) dd[0] = dd[1] = dd[2] = dd[3] = 0.f;
                mma_16816(dd, a0, a1, a2, a3, b[h][0], b[h][1]);
                if (h == 1) {
#pragma unroll
                    for (int e = 0; e < 4; ++e)  // fp8: the 128 x 128 block's fp32 scale multiplies the step's sums
                        c[2 * i + o][e] = MODE == B200MOE_CT_INT8 ? c[2 * i + o][e] + dd[e] : fmaf(sf, dd[e], c[2 * i + o][e]);
                }
            }
        }
    }
}

// fp4: q[0], q[1]: rows (2t, 2t+1) and (2t+8, 2t+9) of the lane's columns 0..7; q[2], q[3]: of its columns 8..15; s0, s1 their
// scales.  The 16 rows are one scale group: the instruction starts from zero and its fp32 sums are multiplied by the group's
// bf16 scale per column into the running totals (the scale never touches a weight; gemv_impl.h:147-199 keeps the weights in fp32
// the same way).
__device__ __forceinline__ void rg_step_fp4(const uint2 (&q)[4], const uint4& s0, const uint4& s1, uint32_t b0, uint32_t b1,
                                            float (&acc)[8][4]) {
    const uint32_t sw[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
    for (int i = 0; i < 2; ++i) {  // columns 8i .. 8i+7 of the lane's 16
        const uint2 lo = q[2 * i], hi = q[2 * i + 1];
        // byte b: the codes of rows (r, r + 1) at column 2b (e_*) / 2b + 1 (o_*)
        const uint32_t e_lo = (lo.x & 0x0F0F0F0Fu) | ((lo.y << 4) & 0xF0F0F0F0u);
        const uint32_t o_lo = ((lo.x >> 4) & 0x0F0F0F0Fu) | (lo.y & 0xF0F0F0F0u);
        const uint32_t e_hi = (hi.x & 0x0F0F0F0Fu) | ((hi.y << 4) & 0xF0F0F0F0u);
        const uint32_t o_hi = ((hi.x >> 4) & 0x0F0F0F0Fu) | (hi.y & 0xF0F0F0F0u);
        uint32_t a0[4], a1[4], a2[4], a3[4];
        cvt_e2m1x8_f16(e_lo, a0);
        cvt_e2m1x8_f16(o_lo, a1);
        cvt_e2m1x8_f16(e_hi, a2);
        cvt_e2m1x8_f16(o_hi, a3);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            float d[4];
            mma_16816_f16_zero(d, a0[b], a1[b], a2[b], a3[b], b0, b1);
            const float sc_e = __uint_as_float(sw[4 * i + b] << 16), sc_o = __uint_as_float(sw[4 * i + b] & 0xFFFF0000u);
            float* c = acc[4 * i + b];
            c[0] = fmaf(d[0], sc_e, c[0]);
            c[1] = fmaf(d[1], sc_e, c[1]);
            c[2] = fmaf(d[2], sc_o, c[2]);
            c[3] = fmaf(d[3], sc_o, c[3]);
        }
    }
}

template <int MODE, bool STORED>
__global__ void __launch_bounds__(kRgThreads, 2)
gemv_ring_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_s,
                 const __grid_constant__ CUtensorMap tmap_x, const GemvArgs a) {
    using T = RgTraits<MODE>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* red = reinterpret_cast<float*>(ring + T::kStages * T::kStageBytes);  // [kKGroups][kRedRows][256]
    RgBarriers* sb = reinterpret_cast<RgBarriers*>(red + T::kKGroups * T::kRedRows * kGvSlabN);
    int* row_start = reinterpret_cast<int*>(sb + 1);
    int* pass_start = row_start + (a.G + 1);  // [G + 1] passes (of up to 8 rows) before the i-th expert

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_slabs = (a.N + kGvSlabN - 1) / kGvSlabN;
    load_row_starts(a.group_list, a.G, a.M, a.gl_type, row_start, a.status);
    if (threadIdx.x < 32) {
        int lo, hi, mine = 0, total, most = 0;
        lane_experts(a.G, lo, hi);
        for (int i = lo; i < hi; ++i) {
            mine += (row_start[i + 1] - row_start[i] + kRgRows - 1) / kRgRows;
            most = max(most, row_start[i + 1] - row_start[i]);
        }
        const int slot_rows = __reduce_max_sync(0xffffffffu, most) > kGvRows ? kRgRows : kGvRows;
        int at = warp_exclusive_sum(mine, total);
        for (int i = lo; i < hi; ++i) {
            pass_start[i] = at;
            at += (row_start[i + 1] - row_start[i] + kRgRows - 1) / kRgRows;
        }
        const int parts = a.part_count == nullptr
                              ? 1
                              : gv_choose_parts((int)min((long long)total * n_slabs, 1LL << 30), gridDim.x, a.K, kGvMaxParts * kGvRows / slot_rows);
        if (threadIdx.x == 0) {
            pass_start[a.G] = total;
            sb->parts = parts;
            sb->slot_rows = slot_rows;
            sb->per_pass = n_slabs * parts;                               // units of one pass
            sb->units = (int)((unsigned)total * (unsigned)sb->per_pass);  // (as many would need 2 TB of y to not fit)
            sb->part_rows = ((a.K + kGvPartRows - 1) / kGvPartRows + parts - 1) / parts * kGvPartRows;
        }
    }
    if (threadIdx.x == 32) {
        sb->abort = 0;
        for (int i = 0; i < T::kStages; ++i) {
            ptx::mbar_init(ptx::smem_u32(&sb->full[i]), 1);
            ptx::mbar_init(ptx::smem_u32(&sb->empty[i]), kRgWarps);
        }
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(ptx::smem_u32(&sb->unit_full[i]), 1);
            ptx::mbar_init(ptx::smem_u32(&sb->unit_empty[i]), kRgWarps);
        }
        ptx::mbar_init(ptx::smem_u32(&sb->sync), kRgWarps);
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tmap_w);
        ptx::prefetch_tensormap(&tmap_x);
        if (T::kFp4) ptx::prefetch_tensormap(&tmap_s);
    }
    __syncthreads();
    grid_dep_wait();  // (the prologue above ran beside the kernel that zeroes the tickets and counters)

    if (warp == kRgWarps) {
        // ------------------------------ producer ------------------------------
        if (lane == 0) {
            const unsigned per_pass = (unsigned)sb->per_pass, units = (unsigned)sb->units;
            uint32_t it = 0, n = 0;  // stages and units handed out
            bool ok = true;
            unsigned held = (unsigned)atomicAdd(a.ticket, 1);
            for (;;) {
                RgUnit u = {};
                const bool live = held < units;
                if (live) {
                    const unsigned pass_no = held / per_pass;
                    int lo = 0, hi = a.G;  // largest expert whose first pass is at most pass_no
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if ((unsigned)pass_start[mid] <= pass_no) lo = mid;
                        else hi = mid;
                    }
                    // expert-major order: the CTAs that run at the same time hold neighbouring slabs of the same experts and
                    // walk the same k rows together, so whole rows of the weight matrix are fetched close in time;
                    // the passes of a slab are adjacent, so all but the first find its weights in L2
                    const unsigned passes = (unsigned)(pass_start[lo + 1] - pass_start[lo]), in = held - (unsigned)pass_start[lo] * per_pass;
                    const unsigned j = in / passes, pass = in - j * passes;
                    const int split = (int)(j / (unsigned)n_slabs), slab = (int)j - split * n_slabs, parts = sb->parts;
                    u.g = lo;
                    u.n0 = slab * kGvSlabN;
                    u.r0 = row_start[lo] + (int)pass * kRgRows;
                    u.rows = min(kRgRows, row_start[lo + 1] - u.r0);
                    u.split = split;
                    u.n_split = parts;
                    u.slot = parts > 1 ? ((pass_start[lo] + (int)pass) * n_slabs + slab) * parts : 0;
                    u.k0 = split * sb->part_rows;
                    u.k1 = min(u.k0 + sb->part_rows, a.K);
                    if constexpr (T::kFp4) {
                        // the fp32 kernel does every four rows (from the expert's first on) of which one is not exact in f16
                        bool all_again = true;
                        for (int q = 0; q < u.rows && all_again; q += kGvRows) {
                            bool bad = false;
                            for (int m = q; m < min(q + kGvRows, u.rows); ++m) bad = bad || __ldca(a.xexp + u.r0 + m) == kGvNotF16;
                            all_again = bad;
                        }
                        if (all_again) {
                            held = (unsigned)atomicAdd(a.ticket, 1);
                            continue;
                        }
                    }
                }
                if (n >= 2 && !rg_wait(&sb->unit_empty[n & 1], ((n >> 1) & 1) ^ 1, sb, a.status, 70)) break;
                sb->unit[n & 1] = u;
                ptx::mbar_arrive(ptx::smem_u32(&sb->unit_full[n & 1]));
                ++n;
                if (!live) break;
                const bool upper = T::kFp4 || u.n0 + 128 < a.N;  // (fp8: the last slab may hold 128 columns)
                for (int k = u.k0; k < u.k1; k += kRgK, ++it) {
                    // The next ticket is drawn when the ring has been filled twice (or with the last stage).  Drawn with the first stage, a CTA
                    // that starts a few us late -- behind the one CTA a row that prepares fp4's x -- found the units of a single wave taken by
                    // others as their second; drawn with the last, two even waves became three on some CTAs.  First stage | twice the ring | last
                    // stage, us: stored fp4, 16 experts of 2 rows, 7168 x 2048, 256 units: 85.9 | 54.9 | 55.0; fp8, 5 tokens x 8, 7168 x 4096, 592 units:
                    // 226 | 226 | 267.
                    if (k == min(u.k0 + 2 * T::kStages * kRgK, (u.k1 - 1) / kRgK * kRgK)) held = (unsigned)atomicAdd(a.ticket, 1);
                    const uint32_t s = it % T::kStages, ph = (it / T::kStages) & 1;
                    if (it >= T::kStages && !rg_wait(&sb->empty[s], ph ^ 1, sb, a.status, 10 + (int)s)) { ok = false; break; }
                    const uint32_t bar = ptx::smem_u32(&sb->full[s]), at = ptx::smem_u32(ring + s * T::kStageBytes);
                    ptx::mbar_arrive_expect_tx(bar, (uint32_t)(upper ? T::kStageBytes : T::kStageBytes - T::kWBytes / 2));
                    if constexpr (T::kFp4) {
                        ptx::tma_load_2d(at, &tmap_w, bar, u.n0 / 2, u.g * a.K + k);
                        ptx::tma_load_2d(at + T::kWBytes, &tmap_s, bar, u.n0, (u.g * a.K + k) / 16);
                    } else {
                        ptx::tma_load_2d(at, &tmap_w, bar, u.n0, u.g * a.K + k);
                        if (upper) ptx::tma_load_2d(at + T::kWBytes / 2, &tmap_w, bar, u.n0 + 128, u.g * a.K + k);
                    }
                    ptx::tma_load_2d(at + T::kWBytes + T::kSBytes, &tmap_x, bar, k, u.r0);
                }
                if (!ok) break;
            }
            if (*reinterpret_cast<volatile int*>(&sb->abort))  // copies in flight land before the shared memory goes
                for (uint32_t j = (it > T::kStages ? it - T::kStages : 0); j < it; ++j)
                    (void)ptx::mbar_wait(ptx::smem_u32(&sb->full[j % T::kStages]), (j / T::kStages) & 1);
        }
        return;
    }

    // ------------------------------ consumers ------------------------------
    const int g = lane >> 2, t = lane & 3, hc = warp % (kRgWarps / T::kKGroups), kg = warp / (kRgWarps / T::kKGroups);
    const int c_warp = hc * T::kCols, kl = kg * T::kKRows;  // the warp's first column in a slab, first k row in a stage
    // the lane's places in a stage; its first column
    const int c_first = c_warp + (!T::kFp4 ? 8 * g : STORED ? 32 * (g >> 2) + 8 * (g & 3) : 16 * g);
    uint32_t w_at[2];
    if constexpr (T::kFp4 && STORED) {
        // stored order: row (b * 4 + aa) * 8 + p of a 64-row block, bytes 32 q ..: four rows' codes of eight columns
        w_at[0] = (uint32_t)((kg * 8 + 4 * hc + (g >> 2)) * 128 + (g & 3) * 32 + 8 * t);
        w_at[1] = w_at[0] + 4 * 8 * 128;  // b = 1: rows 8 .. 15 of the scale group
    } else {
        // 16-byte pieces of a 128-byte row (fp4: of its 256 columns; else of 128), swizzled with the row
        const int row = kl + 2 * t, piece = T::kFp4 ? 4 * hc + (g >> 1) : 4 * (hc & 1) + (g >> 1);
        const int box = T::kFp4 ? 0 : (hc >> 1) * (T::kWBytes / 2);
        w_at[0] = (uint32_t)(box + row * 128 + ((piece ^ (2 * t)) << 4) + (g & 1) * 8);
        w_at[1] = (uint32_t)(box + (row + 1) * 128 + ((piece ^ (2 * t + 1)) << 4) + (g & 1) * 8);
    }
    const uint32_t x_row = (uint32_t)(T::kWBytes + T::kSBytes + g * 128 + 4 * t);
    uint32_t x_at[T::kKRows / 8];  // the lane's words of x row g, 8 k apart
#pragma unroll
    for (int i = 0; i < T::kKRows / 8; ++i) x_at[i] = x_row + (uint32_t)(((kl / 8 + i) ^ g) << 4);
    const uint32_t s_at = (uint32_t)(T::kWBytes + kg * (kGvSlabN * 2) + c_first * 2);
    const uint32_t ring_u32 = ptx::smem_u32(ring);
    const bool sums = MODE == B200MOE_CT_INT8 && a.offset != nullptr;

    uint32_t s = 0, ph = 0, sync_ph = 0;
    for (uint32_t n = 0;; ++n) {
        if (!__all_sync(0xffffffffu, rg_wait(&sb->unit_full[n & 1], (n >> 1) & 1, sb, a.status, 72))) break;
        const RgUnit u = sb->unit[n & 1];
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&sb->unit_empty[n & 1]));
        if (u.rows == 0) break;
        float c[T::kAcc][4];
#pragma unroll
        for (int j = 0; j < T::kAcc; ++j) c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
        // int8: a step's sums are added in fp32 to `run`, and kRgRun steps' to `c`.  The instruction's own additions drop bits: chained over the whole
        // of k they showed two to five times the error of the fp32 multiply-adds that one-row units had before the ring (sums that
        // cancel, 32 experts, 7168 x 4096: 1.1e-7 then, 5.6e-7 chained, 1.1e-7 so; with several rows 2.3e-7 before, 1.0e-7 now), and one
        // level of additions twice.  (32 tokens x 8 over 256 experts, 7168 x 4096: 710 -> 732 us.)
        float run[MODE == B200MOE_CT_INT8 ? T::kAcc : 1][4];
        if constexpr (MODE == B200MOE_CT_INT8) {
#pragma unroll
            for (int j = 0; j < T::kAcc; ++j) run[j][0] = run[j][1] = run[j][2] = run[j][3] = 0.f;
        }
        float xs = 0.f;
        const bool x_on = g < u.rows, cols_on = u.n0 + c_warp < a.N;
        bool ok = true;
        // fp8: the scale of the block (128 k rows: two stages; a part starts with one) is read a block ahead
        const float* sf_at = nullptr;
        float sf = 1.f, sf_next = 1.f;
        if constexpr (MODE == B200MOE_CT_FP8)
            if (cols_on) {
                sf_at = static_cast<const float*>(a.scale) + ((size_t)u.g * (a.K >> 7) + (u.k0 >> 7)) * (a.N >> 7) + ((u.n0 + c_warp) >> 7);
                sf_next = __ldg(sf_at);
            }
        for (int k = u.k0; k < u.k1;) {
            const int k_end = MODE == B200MOE_CT_INT8 ? min(k + kRgRun * kRgK, u.k1) : u.k1;
            for (; k < k_end; k += kRgK) {
                if constexpr (MODE == B200MOE_CT_FP8)
                    if (cols_on && (k & kRgK) == 0) {
                        sf = sf_next;
                        sf_at += a.N >> 7;
                        if (k + 2 * kRgK < u.k1) sf_next = __ldg(sf_at);
                    }
                ok = __all_sync(0xffffffffu, rg_wait(&sb->full[s], ph, sb, a.status, 40 + (int)s));
                if (!ok) break;
                const uint32_t at = ring_u32 + s * T::kStageBytes;
                if (cols_on) {
                    uint32_t b[T::kKRows / 16][2] = {};
                    if (x_on) {
#pragma unroll
                        for (int i = 0; i < T::kKRows / 8; ++i) b[i / 2][i % 2] = lds32(at + x_at[i]);
                    }
                    if constexpr (T::kFp4) {
                        uint2 q[4];
                        if constexpr (STORED) {
#pragma unroll
                            for (int i = 0; i < 2; ++i)
#pragma unroll
                                for (int b = 0; b < 2; ++b) q[2 * i + b] = lds64(at + w_at[b] + i * 256);
                        } else {
                            const uint2 r0w = lds64(at + w_at[0]), r1w = lds64(at + w_at[1]);
                            const uint2 r8w = lds64(at + w_at[0] + 1024), r9w = lds64(at + w_at[1] + 1024);
                            q[0] = make_uint2(r0w.x, r1w.x);
                            q[1] = make_uint2(r8w.x, r9w.x);
                            q[2] = make_uint2(r0w.y, r1w.y);
                            q[3] = make_uint2(r8w.y, r9w.y);
                        }
                        rg_step_fp4(q, lds128(at + s_at), lds128(at + s_at + (STORED ? 128 : 16)), b[0][0], b[0][1], c);
                    } else {
                        if constexpr (MODE == B200MOE_CT_INT8) {
                            rg_step_bytes<MODE>(at + w_at[0], at + w_at[1], b, sf, run);
                        } else {
                            rg_step_bytes<MODE>(at + w_at[0], at + w_at[1], b, sf, c);
                        }
                        if (sums && hc == 0) {
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                xs += (__uint_as_float(b[h][0] << 16) + __uint_as_float(b[h][0] & 0xFFFF0000u)) +
                                      (__uint_as_float(b[h][1] << 16) + __uint_as_float(b[h][1] & 0xFFFF0000u));
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&sb->empty[s]));
                if (++s == T::kStages) { s = 0; ph ^= 1u; }
            }
            if (!ok) break;
            if constexpr (MODE == B200MOE_CT_INT8) {
#pragma unroll
                for (int j = 0; j < T::kAcc; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        c[j][e] += run[j][e];
                        run[j][e] = 0.f;
                    }
            }
        }
        if (!ok) break;

        // ---- the k groups' sums -> shared memory -> one thread per column ----
        if (sums && hc == 0) {
            xs += __shfl_xor_sync(0xffffffffu, xs, 1);
            xs += __shfl_xor_sync(0xffffffffu, xs, 2);
            if (t == 0) sb->xsum[kg][g] = xs;  // (read between the two barriers below)
        }
        const int col = threadIdx.x;
        float v[kRgRows], xv[kRgRows];
#pragma unroll
        for (int m = 0; m < kRgRows; ++m) v[m] = xv[m] = 0.f;
#pragma unroll
        for (int r = 0; r < kRgRows; r += T::kRedRows) {
            if (r < u.rows) {
                if (2 * t >= r && 2 * t < r + T::kRedRows) {
#pragma unroll
                    for (int j = 0; j < T::kAcc; ++j) {
                        const int cc = T::kFp4 && STORED ? c_first + 64 * (j >> 2) + 2 * (j & 3) : c_first + 2 * j;
#pragma unroll
                        for (int e = 0; e < 2; ++e)  // rows 2t, 2t + 1
                            *reinterpret_cast<float2*>(red + (kg * T::kRedRows + 2 * t - r + e) * kGvSlabN + cc) = make_float2(c[j][e], c[j][2 + e]);
                    }
                }
                if (!rg_sync(sb, sync_ph, a.status)) return;
#pragma unroll
                for (int m = 0; m < T::kRedRows; ++m) {
                    if (r + m >= u.rows) break;
#pragma unroll
                    for (int w = 0; w < T::kKGroups; ++w) {
                        v[r + m] += red[(w * T::kRedRows + m) * kGvSlabN + col];
                        if (sums) xv[r + m] += sb->xsum[w][r + m];
                    }
                }
                if (!rg_sync(sb, sync_ph, a.status)) return;
            }
        }

        // ---- a slab in parts: the CTA that arrives last adds them in their order ----
        if (u.n_split > 1) {
            const int slot_rows = sb->slot_rows, slot_floats = slot_rows == kGvRows ? kGvSlotFloats : kRgSlotFloats;
            float* slot = a.part_sums + (size_t)(u.slot + u.split) * slot_floats;
#pragma unroll
            for (int m = 0; m < kRgRows; ++m)
                if (m < u.rows) {
                    __stcg(slot + m * kGvSlabN + col, v[m]);
                    if (sums && col == 0) __stcg(slot + slot_rows * kGvSlabN + m, xv[m]);
                }
            __threadfence();
            if (!rg_sync(sb, sync_ph, a.status)) return;
            if (threadIdx.x == 0) sb->last = atomicAdd(a.part_count + u.slot, 1u) == (unsigned)(u.n_split - 1);
            if (!rg_sync(sb, sync_ph, a.status)) return;
            if (!*reinterpret_cast<volatile int*>(&sb->last)) continue;
            __threadfence();
            if (threadIdx.x == 0) a.part_count[u.slot] = 0u;  // (fp4: the fp32 kernel behind this one counts there too)
            const float* first = a.part_sums + (size_t)u.slot * slot_floats;
#pragma unroll
            for (int m = 0; m < kRgRows; ++m)
                if (m < u.rows) {
                    v[m] = xv[m] = 0.f;
                    for (int p = 0; p < u.n_split; ++p) {
                        v[m] += __ldcg(first + (size_t)p * slot_floats + m * kGvSlabN + col);
                        if (sums) xv[m] += __ldcg(first + (size_t)p * slot_floats + slot_rows * kGvSlabN + m);
                    }
                }
        }
        const int col_y = u.n0 + col;
        if (col_y >= a.N) continue;  // (fp8 only: the upper half of a 128-column last slab)
        float s_n = 1.f, so_n = 0.f;
        if constexpr (MODE == B200MOE_CT_INT8) {
            s_n = __bfloat162float(static_cast<const __nv_bfloat16*>(a.scale)[(size_t)u.g * a.N + col_y]);
            if (sums) so_n = s_n * __bfloat162float(a.offset[(size_t)u.g * a.N + col_y]);
        }
#pragma unroll
        for (int m = 0; m < kRgRows; ++m)
            if (m < u.rows) {
                float o = v[m];
                if constexpr (MODE == B200MOE_CT_INT8) o = fmaf(so_n, xv[m], s_n * (kS8Unit * o));
                if constexpr (T::kFp4) {
                    const int ex = __ldca(a.xexp + u.r0 + m);
                    o = scalbnf(o, ex == kGvNotF16 ? 0 : ex);
                }
                a.y[(size_t)(u.r0 + m) * a.N + col_y] = __float2bfloat16_rn(o);
            }
    }
}

template <int MODE, bool STORED = false>
static int gv_ring_launch(const GemvArgs& a0, cudaStream_t stream) {
    using T = RgTraits<MODE>;
    GemvArgs a = a0;
    a.ticket = a.status + 2;
    CUtensorMap tw, ts, tx;
    int rc = make_tensor_map_2d(&tw, a.weight, 1, (uint64_t)a.G * a.K, T::kFp4 ? a.N / 2 : a.N, kRgK, 128, !(T::kFp4 && STORED));
    if (rc != B200MOE_OK) return rc;
    ts = tw;
    if (T::kFp4) rc = make_tensor_map_2d(&ts, a.scale, 2, (uint64_t)a.G * a.K / 16, a.N, kRgK / 16, kGvSlabN, false);
    if (rc != B200MOE_OK) return rc;
    rc = make_tensor_map_2d(&tx, T::kFp4 ? static_cast<const void*>(a.x16) : a.x, 2, (uint64_t)a.M, a.K, kRgRows, 64, true);
    if (rc != B200MOE_OK) return rc;
    const size_t smem = 1024 + (size_t)T::kStages * T::kStageBytes + sizeof(float) * T::kKGroups * T::kRedRows * kGvSlabN +
                        sizeof(RgBarriers) + sizeof(int) * 2 * (size_t)(a.G + 1);
    B200MOE_CUDA_TRY(cudaFuncSetAttribute(gemv_ring_kernel<MODE, STORED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    B200MOE_CUDA_TRY(launch_dependent(gemv_ring_kernel<MODE, STORED>, 2u * (unsigned)sm_count(), kRgThreads, smem, stream, tw, ts, tx, a));
    return B200MOE_OK;
}

}  // namespace b200moe
