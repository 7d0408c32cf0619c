// Grouped GEMV for decode-sized expert batches (HBM-bandwidth kernels).
//
// Work unit = (up to 4 or 8 rows of a non-empty expert, slab of 256 output columns, part of the k range);
// persistent CTAs draw units from a ticket counter, the passes of a slab next to one another (their weights are then read from L2),
// then the slabs.  K is cut into parts only when whole columns would leave the chip idle (gv_choose_parts); the parts' fp32 sums meet
// in the workspace and the CTA that finishes a slab last adds them up in a fixed order.  Scale and offset are applied in
// the fp32 epilogue and the result is rounded to bf16 once.
// Two kernels.  int8, fp8 and fp4 run on the tensor core with their operands streamed through shared memory (gemv_ring.cuh).  int4, and
// the fp4 rows whose x is not exact in f16, run on fp32 multiply-adds (this file, two CTAs per SM): the unit's x rows are copied to
// shared memory, every warp streams its share of the k rows straight from global memory with coalesced loads, eight row pairs
// in flight before the first is consumed, decodes the packed weights in registers and accumulates with packed two-wide FMAs; the
// 16 half-warp partial sums per column are combined with one shuffle and one pass through shared memory.
#include <algorithm>

#include <cuda_fp16.h>

#include <cstdlib>

#include "common.cuh"

namespace b200moe {

constexpr int kGvSlabN = 256;
constexpr int kGvWarps = 8;
constexpr int kGvThreads = kGvWarps * 32;
constexpr int kGvUnroll = 8;                            // row pairs in flight per lane
constexpr int kGvWarpRows = 2 * kGvUnroll;              // k rows a warp consumes per step
constexpr int kGvIterRows = kGvWarps * kGvWarpRows;     // k rows a CTA consumes per step
constexpr int kGvRows = 4;                              // x rows per pass
constexpr int kGvXPad = 16;                             // bf16 elements between staged x rows (bank spread)

struct GemvArgs {
    const __nv_bfloat16* x;
    const uint8_t* weight;
    const void* scale;
    const __nv_bfloat16* offset;
    const int64_t* group_list;
    __nv_bfloat16* y;
    int M, K, N, G, gl_type;
    int* status;
    int fp4_stored;  // fp4 weights in the reference's pre-shuffled order, read in place
    const __half* x16;  // fp4: x as scaled f16 and the rows' exponents (gv_fp4_prepare_x_kernel), or null: fp32 path only
    const int* xexp;
    unsigned* part_count;  // [kGvMaxParts] finished parts of a slab, zero at the launch; null: k is not split
    float* part_sums;      // [kGvMaxParts][kGvSlotFloats]
    int* ticket;           // status word 2 (the fp32 kernel of fp4: 3, from 1 on)
    int by_rows;           // experts in the order of their row counts: shared memory has room for the order
};

// Split of the k range: parts are multiples of kGvPartRows rows, at most kGvMaxParts of them per launch (four waves of
// two CTAs on 148 SMs; 4.9 MB of partial sums), each with the sums of 4 rows x 256 columns and of the x rows; the tensor-core kernel
// takes two such slots a part where its units have more than four rows.
constexpr int kGvPartRows = 128;
constexpr int kGvMaxParts = 1184;
constexpr int kGvSlotFloats = kGvRows * kGvSlabN + 16;

struct GvUnit {
    int g, r0, rows, n0;  // expert, first row, rows (1 .. kGvRows), first column
    int k0, k1;           // its part of the k range
    int split, n_split;
    int slot;             // first slot of the slab's parts; also its counter
};

typedef unsigned long long f32x2;  // two packed fp32 (sm_100 two-wide FP32 instructions)

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ uint2 ldg_stream8(const uint8_t* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// Decode the lane's 16 columns of one weight row into eight fp32 pairs.
template <int MODE, bool kScaleFp4 = true>
__device__ __forceinline__ void gv_decode(const uint4& q, f32x2 (&w)[8], const f32x2 (&sc)[8], const f32x2 (&tc)[8]) {
    if constexpr (MODE == B200MOE_CT_INT4) {
        // (w + o) * s = w * s + o * s in fp32: sc holds s, tc holds o * s of the row's 128-k group
        const uint32_t w2[2] = {q.x ^ 0x88888888u, q.y ^ 0x88888888u};  // nibble + 8
        const f32x2 kneg = pack2(-8388616.0f, -8388616.0f);             // -(2^23 + 8)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t word = w2[i >> 2];
            const int sh = 8 * (i & 3);
            const float f0 = __uint_as_float(((word >> sh) & 0xFu) | 0x4B000000u);
            const float f1 = __uint_as_float(((word >> (sh + 4)) & 0xFu) | 0x4B000000u);
            w[i] = fma2(add2(pack2(f0, f1), kneg), sc[i], tc[i]);
        }
    } else {  // FP4: q.x, q.y hold 16 codes; per-column scale of the current 16-row group
        const uint32_t w2[2] = {q.x, q.y};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            uint32_t o[4];
            e2m1x8_to_bf16(w2[i], o);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if constexpr (kScaleFp4)
                    w[4 * i + j] = mul2(pack2(__uint_as_float(o[j] << 16), __uint_as_float(o[j] & 0xFFFF0000u)), sc[4 * i + j]);
                else
                    w[4 * i + j] = pack2(__uint_as_float(o[j] << 16), __uint_as_float(o[j] & 0xFFFF0000u));
        }
    }
}

// Takes the CTA's next ticket when the weights of a unit are through: its latency then runs beside the sums.  (Drawn
// earlier, a CTA would sit on a unit while others are idle at the end of the launch.)
__device__ __forceinline__ void gv_draw(const GemvArgs& a, int& next) {
    if (threadIdx.x == 0) next = atomicAdd(a.ticket, 1);
}

// End of a unit: v[m] is the thread's column (threadIdx.x of the slab) of row m summed over the unit's part of k.
// A slab in one part is stored at once.  Otherwise the sums go to the part's slot and the CTA that arrives last adds
// the parts in their order, so the result does not depend on which one that is.
__device__ __forceinline__ void gv_finish(const GemvArgs& a, GvUnit& u, float (&v)[kGvRows]) {
    const int t = threadIdx.x, n = u.n0 + t;
    if (u.n_split > 1) {
        float* slot = a.part_sums + (size_t)(u.slot + u.split) * kGvSlotFloats;
#pragma unroll
        for (int m = 0; m < kGvRows; ++m)
            if (m < u.rows) __stcg(slot + m * kGvSlabN + t, v[m]);
        __threadfence();
        __syncthreads();
        if (t == 0) u.split = atomicAdd(a.part_count + u.slot, 1u) == (unsigned)(u.n_split - 1) ? -1 : 0;  // (no longer needed)
        __syncthreads();
        if (u.split != -1) return;
        __threadfence();
        const float* first = a.part_sums + (size_t)u.slot * kGvSlotFloats;
#pragma unroll
        for (int m = 0; m < kGvRows; ++m) {
            if (m < u.rows) {
                v[m] = 0.f;
                for (int p = 0; p < u.n_split; ++p) v[m] += __ldcg(first + (size_t)p * kGvSlotFloats + m * kGvSlabN + t);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < kGvRows; ++m)
        if (m < u.rows) a.y[(size_t)(u.r0 + m) * a.N + n] = __float2bfloat16_rn(v[m]);
}

template <int MODE, int MB>
__device__ __forceinline__ void gv_compute(const GemvArgs& a, GvUnit& un, const __nv_bfloat16* xs, float* red, int& next) {
    const int g = un.g, n0 = un.n0, k_begin = un.k0, k_end = un.k1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int half = lane >> 4, l16 = lane & 15;
    const size_t row_bytes = (size_t)a.N / 2;
    const uint8_t* wbase = a.weight + (size_t)g * a.K * row_bytes + n0 / 2 + l16 * 8;  // 16 columns per lane
    const int col0 = n0 + l16 * 16;

    f32x2 acc[MB][8];
#pragma unroll
    for (int m = 0; m < MB; ++m)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[m][c] = 0ull;

    f32x2 sc[8], tc[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) sc[c] = tc[c] = 0ull;

    for (int k0 = k_begin + warp * kGvWarpRows; k0 < k_end; k0 += kGvIterRows) {
        // ---- issue all loads of this step first ----
        uint4 q[kGvUnroll];
        const uint8_t* p = wbase + (size_t)(k0 + half) * row_bytes;
#pragma unroll
        for (int u = 0; u < kGvUnroll; ++u) {
            const uint2 v = ldg_stream8(p + (size_t)(2 * u) * row_bytes);
            q[u] = make_uint4(v.x, v.y, 0u, 0u);
        }
        // ---- x values of the 16 rows: lane uses rows k0 + 2u + half ----
        uint32_t xw[MB][kGvUnroll];
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            const uint4* xp = reinterpret_cast<const uint4*>(xs + (size_t)m * (a.K + kGvXPad) + k0);
            const uint4 x0 = xp[0], x1 = xp[1];
            xw[m][0] = x0.x; xw[m][1] = x0.y; xw[m][2] = x0.z; xw[m][3] = x0.w;
            xw[m][4] = x1.x; xw[m][5] = x1.y; xw[m][6] = x1.z; xw[m][7] = x1.w;
        }
        if constexpr (MODE == B200MOE_CT_FP4) {
            // one scale row per 16 k rows: exactly the rows of this step
            const uint4* sp = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.scale) +
                                                             ((size_t)g * (a.K >> 4) + (k0 >> 4)) * a.N + col0);
            const uint4 s0 = __ldg(sp), s1 = __ldg(sp + 1);
            const uint32_t sw[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
            for (int c = 0; c < 8; ++c) sc[c] = pack2(__uint_as_float(sw[c] << 16), __uint_as_float(sw[c] & 0xFFFF0000u));
        } else if constexpr (MODE == B200MOE_CT_INT4) {
            // one scale / offset row per 128 k rows; the 16 rows of this step lie inside one group
            const size_t so = ((size_t)g * (a.K >> 7) + (k0 >> 7)) * a.N + col0;
            const uint4* sp = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.scale) + so);
            const uint4 s0 = __ldg(sp), s1 = __ldg(sp + 1);
            uint4 o0 = make_uint4(0u, 0u, 0u, 0u), o1 = o0;
            if (a.offset != nullptr) {
                const uint4* op = reinterpret_cast<const uint4*>(a.offset + so);
                o0 = __ldg(op);
                o1 = __ldg(op + 1);
            }
            const uint32_t sw[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
            const uint32_t ow[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                sc[c] = pack2(__uint_as_float(sw[c] << 16), __uint_as_float(sw[c] & 0xFFFF0000u));
                tc[c] = mul2(pack2(__uint_as_float(ow[c] << 16), __uint_as_float(ow[c] & 0xFFFF0000u)), sc[c]);
            }
        }
        // fp4 with one or two rows: the step's rows are one scale group, so the scale multiplies the fp32
        // sum of the step's products (x * e2m1 is exact in fp32) instead of every weight
        constexpr bool kGroupScale = (MODE == B200MOE_CT_FP4) && MB <= 2;
        f32x2 part[kGroupScale ? MB : 1][8];
        if constexpr (kGroupScale) {
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int c = 0; c < 8; ++c) part[m][c] = 0ull;
        }
#pragma unroll
        for (int u = 0; u < kGvUnroll; ++u) {
            f32x2 w[8];
            gv_decode<MODE, !kGroupScale>(q[u], w, sc, tc);
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                const float xv = __uint_as_float(half ? (xw[m][u] & 0xFFFF0000u) : (xw[m][u] << 16));
                const f32x2 xx = pack2(xv, xv);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    if constexpr (kGroupScale) part[m][c] = fma2(xx, w[c], part[m][c]);
                    else acc[m][c] = fma2(xx, w[c], acc[m][c]);
                }
            }
        }
        if constexpr (kGroupScale) {
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[m][c] = fma2(part[m][c], sc[c], acc[m][c]);
        }
    }

    // ---- combine the 16 partial sums per column -------------------------------------------------
#pragma unroll
    for (int m = 0; m < MB; ++m) {
        float v[16];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            unpack2(acc[m][c], v[2 * c], v[2 * c + 1]);
            v[2 * c] += __shfl_xor_sync(0xffffffffu, v[2 * c], 16);
            v[2 * c + 1] += __shfl_xor_sync(0xffffffffu, v[2 * c + 1], 16);
        }
        if (half == 0) {
            float4* dst = reinterpret_cast<float4*>(red + ((warp * kGvRows + m) * kGvSlabN) + l16 * 16);
#pragma unroll
            for (int c = 0; c < 4; ++c) dst[c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        }
    }
    gv_draw(a, next);
    __syncthreads();
    float v[kGvRows];
#pragma unroll
    for (int m = 0; m < kGvRows; ++m) {
        v[m] = 0.f;
        if (m < un.rows) {
#pragma unroll
            for (int w = 0; w < kGvWarps; ++w) v[m] += red[(w * kGvRows + m) * kGvSlabN + threadIdx.x];
        }
    }
    gv_finish(a, un, v);
}

// Two e4m3 codes in the high bytes of the two 16-bit lanes (low bytes ignored) -> bf16x2, exact:
// exponent and mantissa bits go under the bf16 exponent, times 2^120 (subnormals included).
__device__ __forceinline__ uint32_t e4m3x2_hi_to_bf16(uint32_t t) {
    return mul_bf16x2(((t >> 4) & 0x07F007F0u) | (t & 0x80008000u), 0x7B807B80u);
}

// ---- fp4 weights in the reference's stored (pre-shuffled) order, read in place -----------------
// Canonical row 16a + 8b + c8 of 64-row block R, byte column 128j + 16p + 4q + s lives at
//   ((((((2R + b) * 4 + a) * 8 + p) * J + j) * 4 + q) * 8 + c8) * 4 + s,        J = N / 256,
// so 16 consecutive bytes are four consecutive rows of eight columns.  A lane therefore owns eight
// columns of the 256-column slab (lane = 16-byte chunk of the output row) and, per step, the 16 rows
// of one scale group: four 16-byte loads, one scale vector.  fp32 throughout; the scale of a group
// multiplies the fp32 sum of its 16 products (x * e2m1 is exact in fp32) instead of every weight.
// No conversion pass over the weights.
template <int MB>
__device__ __forceinline__ void gv_compute_fp4_stored(const GemvArgs& a, GvUnit& un, const __nv_bfloat16* xs,
                                                      float* red, int& next) {
    const int g = un.g, n0 = un.n0, k_begin = un.k0, k_end = un.k1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int J = a.N >> 8, j = n0 >> 8, p = lane >> 2, q = lane & 3;
    const uint8_t* wbase = a.weight + (size_t)g * a.K * ((size_t)a.N >> 1) + (size_t)j * 128 + q * 32;
    const size_t p_stride = (size_t)J * 128;  // bytes between consecutive (b, a, p) rows of the stored array
    const int col0 = n0 + lane * 8;

    f32x2 acc[MB][4];
#pragma unroll
    for (int m = 0; m < MB; ++m)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[m][c] = 0ull;

    for (int k0 = k_begin + warp * 16; k0 < k_end; k0 += kGvWarps * 16) {
        const int R = k0 >> 6, aa = (k0 >> 4) & 3;
        uint4 wq[4];  // [2b + h]: rows k0 + 8b + 4h .. + 3
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const uint8_t* ptr = wbase + ((size_t)((2 * R + b) * 4 + aa) * 8 + p) * p_stride;
            wq[2 * b] = ldg_stream(ptr);
            wq[2 * b + 1] = ldg_stream(ptr + 16);
        }
        const uint4 s4 = __ldg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.scale) +
                                                              ((size_t)g * (a.K >> 4) + (k0 >> 4)) * a.N + col0));
        const uint32_t sw[4] = {s4.x, s4.y, s4.z, s4.w};
        f32x2 sc[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) sc[c] = pack2(__uint_as_float(sw[c] << 16), __uint_as_float(sw[c] & 0xFFFF0000u));
        uint32_t xw[MB][8];  // x of the 16 rows, two per word
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            const uint4* xp = reinterpret_cast<const uint4*>(xs + (size_t)m * (a.K + kGvXPad) + k0);
            const uint4 x0 = xp[0], x1 = xp[1];
            xw[m][0] = x0.x; xw[m][1] = x0.y; xw[m][2] = x0.z; xw[m][3] = x0.w;
            xw[m][4] = x1.x; xw[m][5] = x1.y; xw[m][6] = x1.z; xw[m][7] = x1.w;
        }
        // the 16 rows of the step share one scale per column: sum x * e2m1 first (fp32), scale once
        f32x2 part[MB][4];
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) part[m][c] = 0ull;
#pragma unroll
        for (int piece = 0; piece < 4; ++piece) {
            const uint32_t w4[4] = {wq[piece].x, wq[piece].y, wq[piece].z, wq[piece].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = 4 * piece + i;  // 8b + 4h + i within the step
                uint32_t v[4];
                e2m1x8_to_bf16(w4[i], v);
                f32x2 wv[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) wv[c] = pack2(__uint_as_float(v[c] << 16), __uint_as_float(v[c] & 0xFFFF0000u));
#pragma unroll
                for (int m = 0; m < MB; ++m) {
                    const uint32_t xx = xw[m][row >> 1];
                    const float xv = __uint_as_float((row & 1) ? (xx & 0xFFFF0000u) : (xx << 16));
                    const f32x2 x2 = pack2(xv, xv);
#pragma unroll
                    for (int c = 0; c < 4; ++c) part[m][c] = fma2(x2, wv[c], part[m][c]);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[m][c] = fma2(part[m][c], sc[c], acc[m][c]);
    }
    // partial sums of the eight warps -> shared memory -> one thread per column
#pragma unroll
    for (int m = 0; m < MB; ++m) {
        float v[8];
#pragma unroll
        for (int c = 0; c < 4; ++c) unpack2(acc[m][c], v[2 * c], v[2 * c + 1]);
        float4* dst = reinterpret_cast<float4*>(red + ((warp * kGvRows + m) * kGvSlabN) + lane * 8);
        dst[0] = make_float4(v[0], v[1], v[2], v[3]);
        dst[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
    gv_draw(a, next);
    __syncthreads();
    float v[kGvRows];
#pragma unroll
    for (int m = 0; m < kGvRows; ++m) {
        v[m] = 0.f;
        if (m < un.rows) {
#pragma unroll
            for (int w = 0; w < kGvWarps; ++w) v[m] += red[(w * kGvRows + m) * kGvSlabN + threadIdx.x];
        }
    }
    gv_finish(a, un, v);
}


// Operands of the tensor-core kernel (gemv_ring.cuh).  fp4: the scalar paths spend their issue slots on the decode and the FMAs (about 6
// instructions per weight with four rows; the HBM rate leaves room for fewer than 3).  There the x rows are held as f16 --
// each row scaled by a power of two so that its largest element lies in [2^14, 2^15); that path is only
// taken when every element is then exactly representable, so x' * e2m1 products stay exact.  One shift and two logic
// operations put the two rows' codes of a column into one byte, which the conversion instruction turns into
// the f16 pair (row 2t, row 2t+1) the operand register wants.  The row's power of two is undone in the epilogue.
__device__ __forceinline__ void cvt_e2m1x8_f16(uint32_t w, uint32_t (&o)[4]) {
    // byte i of w = two codes -> f16x2 (low nibble in the low half)
    asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %4; cvt.rn.f16x2.e2m1x2 %0, b0; "
        "cvt.rn.f16x2.e2m1x2 %1, b1; cvt.rn.f16x2.e2m1x2 %2, b2; cvt.rn.f16x2.e2m1x2 %3, b3; }"
        : "=r"(o[0]), "=r"(o[1]), "=r"(o[2]), "=r"(o[3])
        : "r"(w));
}

__device__ __forceinline__ void mma_16816_f16_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                   uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// fp4 prepass, one CTA per x row: the row as f16, times 2^-e with e chosen so that its largest element lies in
// [2^14, 2^15), into x16; e into xexp -- or kGvNotF16 when some element is not exactly representable then (more
// than about 2^-32 below the row's largest, a bf16 subnormal, an infinity or a NaN): such rows take the fp32 path.
constexpr int kGvNotF16 = -(1 << 30);

// A row of the second kind also raises status word 3, the ticket of the fp32 kernel, from 0 (nothing to do) to 1.
__global__ void __launch_bounds__(256) gv_fp4_prepare_x_kernel(const __nv_bfloat16* __restrict__ x, __half* __restrict__ x16,
                                                               int* __restrict__ xexp, int K, int* __restrict__ status) {
    grid_dep_launch();
    __shared__ int s_max, s_bad;
    const size_t row = blockIdx.x;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(x + row * K);
    uint32_t* dst = reinterpret_cast<uint32_t*>(x16 + row * K);
    if (threadIdx.x == 0) { s_max = 0; s_bad = 0; }
    __syncthreads();
    uint32_t mx = 0u;
    for (int i = threadIdx.x; i < K / 2; i += blockDim.x) {
        const uint32_t w = __ldg(src + i);
        mx = max(mx, max(w & 0x7FFFu, (w >> 16) & 0x7FFFu));  // bf16 magnitudes order like integers
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&s_max, (int)mx);
    __syncthreads();
    const int e_max = s_max >> 7;                    // biased exponent of the largest magnitude
    const int sh = e_max == 0 ? 0 : e_max - 127 - 14;
    int bad = e_max == 255;
    for (int i = threadIdx.x; i < K / 2; i += blockDim.x) {
        const uint32_t w = __ldg(src + i);
        uint32_t out = 0u;
#pragma unroll
        for (int hlf = 0; hlf < 2; ++hlf) {
            const uint32_t b = hlf ? (w >> 16) : (w & 0xFFFFu);
            const uint32_t mag = b & 0x7FFFu, sign = b & 0x8000u;
            uint32_t h = sign;
            if (mag != 0u) {
                const int e = (int)(mag >> 7);
                const int E = e - sh - 112;                       // biased f16 exponent of the scaled value
                const uint32_t sig = (0x80u | (mag & 0x7Fu)) << 3;  // 11-bit significand, leading one at bit 10
                if (e == 0 || E > 30) bad = 1;
                else if (E >= 1) h = sign | ((uint32_t)E << 10) | (sig & 0x3FFu);
                else {
                    const int s = 1 - E;                          // f16 subnormal: exact only if no set bit is shifted out
                    if (s > 10 || (sig & ((1u << s) - 1u)) != 0u) bad = 1;
                    else h = sign | (sig >> s);
                }
            }
            out |= h << (16 * hlf);
        }
        dst[i] = out;
    }
    if (bad) atomicOr(&s_bad, 1);
    __syncthreads();
    grid_dep_wait();  // (launched beside gv_begin_kernel, which zeroes the status words; what follows this kernel also follows that)
    if (threadIdx.x == 0) {
        xexp[row] = s_bad ? kGvNotF16 : sh;
        if (s_bad) atomicMax(status + 3, 1);
    }
}

// Clears what a call starts from: status words 0 .. 3 and the counters of the k parts (words 4, 5 are the caller's).
__global__ void __launch_bounds__(256) gv_begin_kernel(int* __restrict__ status, unsigned* __restrict__ part_count) {
    grid_dep_launch();
    if (threadIdx.x < 4) status[threadIdx.x] = 0;
    if (part_count != nullptr)
        for (int i = threadIdx.x; i < kGvMaxParts; i += blockDim.x) part_count[i] = 0u;
}

// Parts a slab's k range is cut into, for `slabs` (rows x slab) units on `ctas` CTAs; called by a whole warp, lane i
// weighs i + 1 parts: waves of CTAs times the blocks of kGvPartRows rows of a part plus kGvPartCost, what a unit costs
// beyond its weights (first loads, the sums' way through L2; in grouped_gemv_kernel the staging of x too) in blocks.  A launch of many
// waves has nothing to gain and stays whole.  Whole | in parts, us, register kernel: one token on 8 of 256 experts, 7168 x 4096 fp8 (128
// slabs, two parts): 117 | 72; 3 tokens x 4 over 160 experts, 4224 x 3328 int8: 54.6 | 53.3.  In the ring kernel costs of 1, 2 and 4 give the
// same times (32, 128, 160, 336 and 368 slabs, three formats: within 1 %, fp4 at 32 slabs 5 %): the count of waves decides.
constexpr int kGvPartCost = 2;
__device__ __forceinline__ int gv_choose_parts(int slabs, int ctas, int K, int max_parts) {
    const int blocks = (K + kGvPartRows - 1) / kGvPartRows;
    const int s = (threadIdx.x & 31) + 1, per = (blocks + s - 1) / s;
    unsigned cost = 0xFFFFFFFFu;
    if (s == 1 || ((long long)slabs * s <= max_parts && per > 1 && (blocks + per - 1) / per == s))
        cost = min((unsigned)((slabs * (long long)s + ctas - 1) / ctas) * (unsigned)(per + kGvPartCost), 0x03FFFFFFu) * 32u + (unsigned)(s - 1);
    return (int)(__reduce_min_sync(0xffffffffu, cost) & 31u) + 1;
}

// fp4 is launched as two kernels over the same rows: gemv_ring_kernel, and behind it this one as PATH 1 for the passes of which an x
// row is not exact as scaled f16 (normally none: it leaves at once when the prepass found no such row).
template <int MODE, int PATH = 0>
__global__ void __launch_bounds__(kGvThreads, 2) grouped_gemv_kernel(const GemvArgs a) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    int* row_start = reinterpret_cast<int*>(smem_raw);
    int* pass_start = row_start + (a.G + 1);  // [G + 1] passes (of up to 4 rows) before the i-th expert in order
    int* order = pass_start + (a.G + 1);      // [G], with by_rows
    uintptr_t p = (reinterpret_cast<uintptr_t>(order + (a.by_rows ? a.G : 0)) + 15) & ~uintptr_t(15);
    float* red = reinterpret_cast<float*>(p);                                     // [8][4][256]
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(red + kGvWarps * kGvRows * kGvSlabN);  // [4][K]

    if (PATH == 1) {
        grid_dep_wait();
        if (*reinterpret_cast<volatile int*>(a.status + 3) == 0) return;
    }
    __shared__ GvUnit un;
    __shared__ int s_ticket, s_parts, s_part_rows;
    __shared__ unsigned s_per_pass, s_units;
    const int n_slabs = (a.N + kGvSlabN - 1) / kGvSlabN;
    load_row_starts(a.group_list, a.G, a.M, a.gl_type, row_start, a.status);
    if (threadIdx.x < 32) {
        int lo, hi, mine = 0, total;
        lane_experts(a.G, lo, hi);
        if (a.by_rows) {
            // counting sort on min(rows, 5), the most rows first: units of the same number of rows run together (the
            // row count picks the code path) and the long ones start early.  32 tokens x 8 over 256 experts,
            // 7168 x 4096 int8: 3 % slower in the experts' own order.
            int n = 0;
            for (int b = 5; b >= 0; --b) {
                int same = 0, all;
                for (int g = lo; g < hi; ++g) same += min(row_start[g + 1] - row_start[g], 5) == b;
                int to = n + warp_exclusive_sum(same, all);
                if (all > 0)
                    for (int g = lo; g < hi; ++g)
                        if (min(row_start[g + 1] - row_start[g], 5) == b) order[to++] = g;
                n += all;
            }
            __syncwarp();
        }
        auto passes_of = [&](int i) {
            const int g = a.by_rows ? order[i] : i;
            return (row_start[g + 1] - row_start[g] + kGvRows - 1) / kGvRows;
        };
        for (int i = lo; i < hi; ++i) mine += passes_of(i);
        int at = warp_exclusive_sum(mine, total);
        for (int i = lo; i < hi; ++i) {
            pass_start[i] = at;
            at += passes_of(i);
        }
        if (threadIdx.x == 0) pass_start[a.G] = total;
        const int parts = a.part_count == nullptr ? 1 : gv_choose_parts((int)min((long long)total * n_slabs, 1LL << 30), gridDim.x, a.K, kGvMaxParts);
        if (threadIdx.x == 0) {
            // (kept in shared memory: a unit's loop needs every register)
            s_parts = parts;
            s_per_pass = (unsigned)(n_slabs * parts);  // units of one pass
            s_units = (unsigned)total * s_per_pass;    // (32 bits hold every unit number: y alone would take 2 TB with 2^30 units)
            s_part_rows = ((a.K + kGvPartRows - 1) / kGvPartRows + parts - 1) / parts * kGvPartRows;
        }
    }
    __syncthreads();

    grid_dep_wait();  // (the prologue above ran beside the kernel that zeroes the tickets and counters)
    int next = 0;  // thread 0: the ticket drawn last
    gv_draw(a, next);
    for (;;) {
        if (threadIdx.x == 0) s_ticket = next;
        __syncthreads();
        const unsigned unit = (unsigned)(s_ticket - (PATH == 1 ? 1 : 0));
        if (unit >= s_units) break;
        // every thread looks at its experts, the one that finds the unit describes it to the others: a binary search
        // with its divisions by one thread was a tenth of a short unit (2048 rows of fp4)
        for (int i = threadIdx.x; i < a.G; i += kGvThreads) {
            const unsigned per_pass = s_per_pass, first = (unsigned)pass_start[i] * per_pass, passes = (unsigned)(pass_start[i + 1] - pass_start[i]);
            if (unit < first || unit - first >= passes * per_pass) continue;
            const int g = a.by_rows ? order[i] : i;
            // expert-major order: the CTAs that run at the same time hold neighbouring slabs of the same experts
            // and walk the same k rows together, so whole rows of the weight matrix are fetched close in time
            // (DRAM pages stay open: measured +1..6 % over slab-major order); the passes of a slab are
            // adjacent, so all but the first find its weights in L2
            const unsigned j = (unit - first) / passes, pass = (unit - first) - j * passes;
            const int n_slabs = (a.N + kGvSlabN - 1) / kGvSlabN, n_parts = s_parts;
            const int split = (int)(j / (unsigned)n_slabs), slab = (int)j - split * n_slabs;
            un.g = g;
            un.n0 = slab * kGvSlabN;
            un.r0 = row_start[g] + (int)pass * kGvRows;
            un.rows = min(kGvRows, row_start[g + 1] - un.r0);
            un.split = split;
            un.n_split = n_parts;
            un.slot = n_parts > 1 ? ((pass_start[i] + (int)pass) * n_slabs + slab) * n_parts : 0;
            un.k0 = split * s_part_rows;
            un.k1 = min(un.k0 + s_part_rows, a.K);
        }
        __syncthreads();
        {
            // (copies: the stores of the staging loop could alias the descriptor)
            const int r = un.r0, rows = un.rows, v0 = un.k0 / 8, v1 = un.k1 / 8;
            if constexpr (PATH == 1) {
                bool exact = true;
                for (int m = 0; m < rows; ++m) exact = exact && a.xexp[r + m] != kGvNotF16;
                if (exact) {  // the other kernel's pass
                    gv_draw(a, next);
                    __syncthreads();
                    continue;
                }
            }
            // ---- stage the x rows ----
            for (int m = 0; m < rows; ++m) {
                const uint4* src = reinterpret_cast<const uint4*>(a.x + (size_t)(r + m) * a.K);
                uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)m * (a.K + kGvXPad));
#pragma unroll 4
                for (int i = v0 + threadIdx.x; i < v1; i += kGvThreads) {
                    const uint4 v = PATH == 1 ? __ldca(src + i) : __ldg(src + i);
                    dst[i] = v;
                }
            }
            __syncthreads();
            if (MODE == B200MOE_CT_FP4 && a.fp4_stored) {
                if (rows == 1) gv_compute_fp4_stored<1>(a, un, xs, red, next);
                else if (rows == 2) gv_compute_fp4_stored<2>(a, un, xs, red, next);
                else gv_compute_fp4_stored<4>(a, un, xs, red, next);
            } else if (rows == 1) gv_compute<MODE, 1>(a, un, xs, red, next);
            else if (rows == 2) gv_compute<MODE, 2>(a, un, xs, red, next);
            else gv_compute<MODE, 4>(a, un, xs, red, next);
        }
    }
}

constexpr size_t kGvSmemLimit = 227 * 1024;
static size_t gv_smem_bytes(int G, int K, bool by_rows) {
    size_t b = (sizeof(int) * (size_t)((by_rows ? 3 : 2) * G + 2) + 15) & ~size_t(15);
    b += sizeof(float) * kGvWarps * kGvRows * kGvSlabN;
    b += ((size_t)kGvRows * K + (kGvRows - 1) * kGvXPad) * 2;
    return b;
}

template <int MODE, int PATH = 0>
static int gv_launch(const GemvArgs& a0, cudaStream_t stream) {
    GemvArgs a = a0;
    a.ticket = a.status + (PATH == 1 ? 3 : 2);
    size_t smem = gv_smem_bytes(a.G, a.K, true);
    // (the order must not cost the second CTA of a multiprocessor, nor a shape that fits without it)
    a.by_rows = smem <= 110 * 1024 || (smem <= 226 * 1024 && gv_smem_bytes(a.G, a.K, false) > 110 * 1024);
    if (!a.by_rows) smem = gv_smem_bytes(a.G, a.K, false);
    // One CTA a multiprocessor: room for exactly one.  A kernel that starts beside the one before it has its CTAs put wherever
    // there is room, and where two fitted, some SMs got two and others none (stored fp4, 16 tokens x 8 over 64 experts,
    // 10240 x 1024, 115 KB: 236 us; 188 with one on each).
    const int per_sm = smem <= 110 * 1024 ? 2 : 1;
    if (per_sm == 1) smem = std::max<size_t>(smem, 116 * 1024);
    B200MOE_CUDA_TRY(cudaFuncSetAttribute(grouped_gemv_kernel<MODE, PATH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
    // (behind gv_begin_kernel, or as PATH 1 behind the tensor-core kernel)
    B200MOE_CUDA_TRY(launch_dependent(grouped_gemv_kernel<MODE, PATH>, (unsigned)(per_sm * sm_count()), kGvThreads, smem, stream, a));
    return B200MOE_OK;
}

}  // namespace b200moe

#include "gemv_ring.cuh"

using namespace b200moe;

constexpr size_t kGvCountBytes = (kGvMaxParts * sizeof(unsigned) + 255) / 256 * 256;
constexpr size_t kGvPartBytes = kGvCountBytes + kGvMaxParts * sizeof(float) * kGvSlotFloats;
static_assert(kGvPartBytes % 256 == 0, "what follows stays aligned");
static size_t gv_fp4_exp_bytes(int64_t M) { return ((size_t)M * sizeof(int) + 255) / 256 * 256; }

extern "C" size_t b200moe_grouped_gemv_workspace_bytes(int64_t M, int64_t K, int64_t N, int64_t G, int compute_type,
                                                       int weight_layout) {
    (void)N; (void)G; (void)weight_layout;
    // status words and the work-unit tickets; fp4 adds the rows' exponents and x as scaled f16
    size_t b = B200MOE_STATUS_BYTES;
    if (compute_type == B200MOE_CT_FP4 && M > 0 && K > 0) b += gv_fp4_exp_bytes(M) + (size_t)M * (size_t)K * 2;
    return b;
}

// ... and, behind that, the counters and sums of the k parts.
static size_t gv_parts_offset(size_t base) { return (base + 255) / 256 * 256; }

extern "C" size_t b200moe_grouped_gemv_split_workspace_bytes(int64_t M, int64_t K, int64_t N, int64_t G, int compute_type,
                                                             int weight_layout) {
    return gv_parts_offset(b200moe_grouped_gemv_workspace_bytes(M, K, N, G, compute_type, weight_layout)) + kGvPartBytes;
}

extern "C" int b200moe_grouped_gemv(const void* x, const void* weight, const void* scale, const void* offset,
                                    const int64_t* group_list, void* y, int64_t M, int64_t K, int64_t N, int64_t G,
                                    int compute_type, int group_list_type, int weight_layout, void* workspace,
                                    size_t workspace_bytes, void* stream) {
    if (compute_type < B200MOE_CT_FP8 || compute_type > B200MOE_CT_INT4) return B200MOE_ERR_COMPUTE_TYPE;
    if (group_list_type != B200MOE_GROUP_LIST_CUMSUM && group_list_type != B200MOE_GROUP_LIST_COUNTS)
        return B200MOE_ERR_ARGUMENT;
    if (weight_layout != B200MOE_LAYOUT_CANONICAL && weight_layout != B200MOE_LAYOUT_ASCEND)
        return B200MOE_ERR_ARGUMENT;
    if (M < 0 || K <= 0 || N <= 0 || G <= 0 || G > kMaxExperts || M > 0x7FFFFFF0LL || K > 0x7FFFFFF0LL ||
        N > 0x7FFFFFF0LL || G * K > 0x7FFFFFF0LL)
        return B200MOE_ERR_SHAPE;
    // fp8: what the reference takes (K and N multiples of its 128 x 128 scale block, i.e. a last slab of
    // 128 columns); the other modes work on whole 256-column slabs
    if (compute_type == B200MOE_CT_FP8 ? ((K % 128) != 0 || (N % 128) != 0) : ((K % 64) != 0 || (N % kGvSlabN) != 0))
        return B200MOE_ERR_SHAPE;
    if (compute_type == B200MOE_CT_INT4 && (K % 128) != 0) return B200MOE_ERR_SHAPE;
    if (M == 0) return B200MOE_OK;
    if (!x || !weight || !scale || !group_list || !y) return B200MOE_ERR_NULL_POINTER;
    if (!aligned16(x) || !aligned16(weight) || !aligned16(scale) || !aligned16(y) ||
        (offset && !aligned16(offset)))
        return B200MOE_ERR_ALIGNMENT;
    const size_t need = b200moe_grouped_gemv_workspace_bytes(M, K, N, G, compute_type, weight_layout);
    if (workspace == nullptr || workspace_bytes < need || !aligned16(workspace)) return B200MOE_ERR_WORKSPACE;
    // (K up to what the fp32 kernels' staged x rows allow: one limit for every format, refused before anything is launched)
    if (gv_smem_bytes((int)G, (int)K, false) > kGvSmemLimit) return B200MOE_ERR_SHAPE;

    cudaStream_t s = static_cast<cudaStream_t>(stream);
    GemvArgs a;
    a.x = static_cast<const __nv_bfloat16*>(x);
    a.weight = static_cast<const uint8_t*>(weight);
    a.scale = scale;
    a.offset = static_cast<const __nv_bfloat16*>(offset);
    a.group_list = group_list;
    a.y = static_cast<__nv_bfloat16*>(y);
    a.M = (int)M; a.K = (int)K; a.N = (int)N; a.G = (int)G;
    a.gl_type = group_list_type;
    a.status = static_cast<int*>(workspace);
    uint8_t* ws = static_cast<uint8_t*>(workspace) + B200MOE_STATUS_BYTES;
    a.part_count = nullptr;
    a.part_sums = nullptr;
    if (workspace_bytes >= gv_parts_offset(need) + kGvPartBytes) {
        uint8_t* parts = static_cast<uint8_t*>(workspace) + gv_parts_offset(need);
        a.part_count = reinterpret_cast<unsigned*>(parts);
        a.part_sums = reinterpret_cast<float*>(parts + kGvCountBytes);
    }
    gv_begin_kernel<<<1, 256, 0, s>>>(a.status, a.part_count);
    B200MOE_CUDA_TRY(cudaGetLastError());

    // fp4 in the stored (pre-shuffled) order is read in place
    a.fp4_stored = (compute_type == B200MOE_CT_FP4 && weight_layout == B200MOE_LAYOUT_ASCEND) ? 1 : 0;
    a.x16 = nullptr;
    a.xexp = nullptr;
    // (B200MOE_GEMV_FP4_SCALAR=1 keeps fp4 on the fp32 multiply-adds: comparison runs)
    static const bool fp4_scalar = [] { const char* e = getenv("B200MOE_GEMV_FP4_SCALAR"); return e && e[0] == '1'; }();
    if (compute_type == B200MOE_CT_FP4 && !fp4_scalar) {
        a.xexp = reinterpret_cast<const int*>(ws);
        a.x16 = reinterpret_cast<const __half*>(ws + gv_fp4_exp_bytes(M));
        // (beside gv_begin_kernel: 8 experts, 4 tokens x 2, 512 x 1024, stored order: 22.6 us one after the other, 20.5 so; a memset
        // in the place of gv_begin_kernel: 21 .. 24)
        B200MOE_CUDA_TRY(launch_dependent(gv_fp4_prepare_x_kernel, (unsigned)M, 256, 0, s, a.x, const_cast<__half*>(a.x16),
                                          const_cast<int*>(a.xexp), a.K, a.status));
    }
    switch (compute_type) {
        case B200MOE_CT_INT8: return gv_ring_launch<B200MOE_CT_INT8>(a, s);
        case B200MOE_CT_FP8: return gv_ring_launch<B200MOE_CT_FP8>(a, s);
        case B200MOE_CT_INT4: return gv_launch<B200MOE_CT_INT4>(a, s);
        default: {
            if (a.x16 == nullptr) return gv_launch<B200MOE_CT_FP4>(a, s);
            const int rc = a.fp4_stored ? gv_ring_launch<B200MOE_CT_FP4, true>(a, s) : gv_ring_launch<B200MOE_CT_FP4, false>(a, s);
            if (rc != B200MOE_OK) return rc;
            return gv_launch<B200MOE_CT_FP4, 1>(a, s);
        }
    }
}
