// Shared device/host helpers of the b200moe kernels (sm_100a only).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/b200moe.h"

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 1000)
#error "b200moe kernels are written for sm_100a"
#endif

namespace b200moe {

// Device status words (first 16 bytes of a workspace).
constexpr int kDevOk = 0;
constexpr int kDevBadGroupList = 1;
constexpr int kDevWaitExpired = 2;

// Records a device-side finding in the status words of a workspace: words 0 / 1 (zeroed by every
// entry point before its launch) hold the code and detail of the current call, words 4 / 5 keep the
// first finding of ANY call that used this workspace since the caller last zeroed them -- a binding
// that reuses one workspace can check them at its own synchronisation points.
__device__ __forceinline__ void report_status(int* status, int code, int detail) {
    if (status == nullptr) return;
    if (atomicCAS(status, 0, code) == 0) status[1] = detail;
    if (atomicCAS(status + 4, 0, code) == 0) status[5] = detail;
}

// Largest expert count the kernels keep in shared memory.
constexpr int kMaxExperts = 1024;

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

#define B200MOE_CUDA_TRY(expr)                      \
    do {                                            \
        cudaError_t e__ = (expr);                   \
        if (e__ != cudaSuccess) {                   \
            (void)cudaGetLastError();               \
            return B200MOE_ERR_CUDA;                \
        }                                           \
    } while (0)

// A kernel launched with launch_dependent may start while the kernel before it in the stream is still running, once all of
// that kernel's blocks have called grid_dep_launch() or ended; grid_dep_wait() returns when it has completed and its
// writes are visible (at once in a kernel launched the usual way).  What that kernel writes is not read-only for the whole
// of this one's lifetime, so it is read with ordinary loads (__ldca, __ldcg), never with __ldg: non-coherent
// loads are defined for data that nothing writes while the kernel is there.
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... Params, class... Args>
inline cudaError_t launch_dependent(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                                    const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// Weights that are read once by this SM: not kept in L1.  (GEMM, 8192 tokens x 8 over 256 experts, 7168 x 4096: int4 9.3 ->
// 9.1 ms, fp8 6.07 -> 5.97; the packed int8 kernel lost 3 % with it, and the fp4 forms share sectors between loads.)
__device__ __forceinline__ uint4 ldg_stream(const uint8_t* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg_stream4(const uint8_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// Multiprocessor count of the current device (cached per device).
int sm_count();

// ---- tensor maps (driver entry point fetched through the runtime, no libcuda link) ---------
// 2-D row-major tensor [rows, cols] of `elem_bytes`-byte elements, box [box_rows, box_cols].
// swizzle128: 128-byte swizzle (box_cols * elem_bytes must be 128), else no swizzle.
int make_tensor_map_2d(CUtensorMap* out, const void* base, int elem_bytes, uint64_t rows, uint64_t cols,
                       uint32_t box_rows, uint32_t box_cols, bool swizzle128);

// ---- small device utilities ---------------------------------------------------------------
__device__ __forceinline__ float bf16_bits_to_float(uint32_t b) { return __uint_as_float(b << 16); }

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// Two fp32 values in one 64-bit register for the two-wide FP32 instructions of sm_100.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack_u32x2(uint32_t lo, uint32_t hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ f32x2 pack_f32x2(float lo, float hi) {
    return pack_u32x2(__float_as_uint(lo), __float_as_uint(hi));
}
__device__ __forceinline__ float f32x2_lo(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float f32x2_hi(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ f32x2 mul_f32x2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub_f32x2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma_f32x2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

// The warp's 16 x 8 += 16 x 16 by 16 x 8 in bf16, sums in fp32.
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Eight packed FP4 e2m1 codes (nibble i = element i) -> eight bf16 values, in element order.
// The three magnitude bits of a code are dropped into bf16 bits [8:6] (two exponent LSBs and the
// mantissa MSB) and the sign into bit 15; read as bf16 that is value * 2^-126 including the subnormal code 0.5, so one
// exact multiply by 2^126 yields the e2m1 value.  Codes i and i+4 sit 16 bits apart and share
// one bf16x2 lane pair.  With the pair's nibbles alone in a word, its copies 6 and 12 bits up do not overlap: one integer
// multiply makes both, on the FMA pipe instead of two shifts on the half-rate ALU pipe, and one mask keeps the bits wanted of either.
// e2m1x8_to_bf16_tiny leaves the pairs that way: out[i] = elements (i, i + 4) times 2^-126.
// (13 instructions per eight codes, and 4 more where the 2^126 rides in the scale, instead of 23: fp4 GEMM of 32 rows an expert,
// 256 experts, 2048 x 7168, 1244 -> 1215 us; fp4-stored layer of 256 experts, 4096 tokens x 8, 4911 -> 4810.)
constexpr uint32_t kTwo126 = 0x7E807E80u;  // bf16x2
__device__ __forceinline__ void e2m1x8_to_bf16_tiny(uint32_t w, uint32_t out[4]) {
    const uint32_t v = w >> 8;
    out[0] = ((w & 0x000F000Fu) * 0x1040u) & 0x81C081C0u;
    out[1] = ((w & 0x00F000F0u) * 0x0104u) & 0x81C081C0u;
    out[2] = ((v & 0x000F000Fu) * 0x1040u) & 0x81C081C0u;
    out[3] = ((v & 0x00F000F0u) * 0x0104u) & 0x81C081C0u;
}
// ... and the values themselves: out[i] = elements (i, i + 4).
__device__ __forceinline__ void e2m1x8_to_bf16_pairs(uint32_t w, uint32_t out[4]) {
    e2m1x8_to_bf16_tiny(w, out);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = mul_bf16x2(out[i], kTwo126);
}
__device__ __forceinline__ void e2m1x8_to_bf16(uint32_t w, uint32_t out[4]) {
    uint32_t r[4];
    e2m1x8_to_bf16_pairs(w, r);
    out[0] = prmt(r[0], r[1], 0x5410);
    out[1] = prmt(r[2], r[3], 0x5410);
    out[2] = prmt(r[0], r[1], 0x7632);
    out[3] = prmt(r[2], r[3], 0x7632);
}

// Four signed int8 (one 32-bit word) -> four bf16 of value / 64, exact, in five instructions (two of them on the FMA pipe;
// seven when the sign bit was taken out by a subtraction: decode layer of 256 experts, 32 tokens x 8, 7168 x 2048, packed GEMMs
// 1592 -> 1561 us, GEMV of the same tokens, 7168 x 4096, 923 -> 899).
// byte ^ 0x80 = value + 128 = p; the bf16 with the bits p (0 .. 255: the subnormals and the first binade, one spacing) is
// p * 2^-133, so one fused multiply-add p * 2^-133 * 2^127 - 2 yields value / 64 without a rounding.  The masks pick bytes 0 and
// 2 of the word (and 1 and 3 after a shift): `o02` holds elements (0, 2), `o13` elements (1, 3).  Whoever sums the
// products multiplies the fp32 sum by kS8Unit.
constexpr float kS8Unit = 64.f;
__device__ __forceinline__ float s8_sum(uint32_t acc) { return kS8Unit * __uint_as_float(acc); }
__device__ __forceinline__ void s8x4_to_bf16_even_odd(uint32_t w, uint32_t& o02, uint32_t& o13) {
    uint32_t p;
    asm("lop3.b32 %0, %1, 0x00FF00FF, 0x00800080, 0x6A;" : "=r"(p) : "r"(w));  // (w & m) ^ c
    o02 = fma_bf16x2(p, 0x7F007F00u, 0xC000C000u);
    asm("lop3.b32 %0, %1, 0x00FF00FF, 0x00800080, 0x6A;" : "=r"(p) : "r"(w >> 8));
    o13 = fma_bf16x2(p, 0x7F007F00u, 0xC000C000u);
}

// Sum over the lanes below this one and, in `total`, over the whole warp.
__device__ __forceinline__ int warp_exclusive_sum(int v, int& total) {
    const int lane = threadIdx.x & 31;
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += n;
    }
    total = __shfl_sync(0xffffffffu, s, 31);
    return s - v;
}

// The consecutive experts a lane of the scheduling warp owns: [lo, hi) of G.
__device__ __forceinline__ void lane_experts(int G, int& lo, int& hi) {
    const int per = (G + 31) >> 5;
    lo = min((int)(threadIdx.x & 31) * per, G);
    hi = min(lo + per, G);
}

// Row boundaries of every expert from the device-side group_list, clamped into [0, M] and made
// monotone so no later index can leave the tensors; a violation is reported in the status words.
// Executed by a whole CTA; row_start has G+1 entries in shared memory.  G <= kMaxExperts.
// Every thread fetches entries, then the first warp scans them, each lane a stretch of consecutive
// experts: with one thread walking the 256 entries, the GEMV of one token (8 rows, 7168 x 4096, fp8) took
// 152 us instead of 110 and that of 37 tokens (2048 x 7168, fp4) 475 instead of 429.
__device__ __forceinline__ void load_row_starts(const int64_t* __restrict__ gl, int G, int M, int gl_type,
                                                int* row_start, int* status) {
    for (int g = threadIdx.x; g < G; g += blockDim.x) {
        const long long v = gl[g];
        row_start[g + 1] = (int)(v < -1 ? -1 : (v > (long long)M + 1 ? (long long)M + 1 : v));
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool counts = gl_type == B200MOE_GROUP_LIST_COUNTS;
        const int lane = threadIdx.x;
        int lo, hi;
        lane_experts(G, lo, hi);
        // what the lane's stretch adds up to: a sum of counts, or the largest boundary (both without the
        // invalid negative entries), saturated at M + 1: beyond M nothing changes any more (M < 2^31, so
        // the sum of two saturated values fits 32 unsigned bits)
        const uint32_t m = (uint32_t)M, cap = m + 1u;
        uint32_t mine = 0;
        for (int g = lo; g < hi; ++g) {
            const uint32_t v = (uint32_t)max(row_start[g + 1], 0);
            mine = counts ? min(mine + v, cap) : max(mine, v);
        }
        uint32_t pre = mine;  // inclusive scan, then shifted by one lane
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t n = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre = counts ? min(pre + n, cap) : max(pre, n);
        }
        pre = __shfl_up_sync(0xffffffffu, pre, 1);
        if (lane == 0) pre = 0;
        int bad_at = G;
        for (int g = lo; g < hi; ++g) {
            const int v = row_start[g + 1];
            const uint32_t end = counts ? pre + (uint32_t)max(v, 0) : (uint32_t)max(v, 0);
            // (after an end beyond M the list stays at M, so a later boundary below M is a step back)
            if (v < 0 || end < min(pre, m) || end > m) bad_at = min(bad_at, g);
            pre = counts ? min(end, cap) : max(pre, end);
            row_start[g + 1] = (int)min(pre, m);
        }
        if (lane == 0) row_start[0] = 0;
        bad_at = __reduce_min_sync(0xffffffffu, bad_at);
        if (lane == 0 && bad_at < G) {
            grid_dep_wait();  // the kernel before this one may still have to zero the status words
            report_status(status, kDevBadGroupList, bad_at);
        }
    }
    __syncthreads();
}

}  // namespace b200moe
