// Arguments shared by the grouped-GEMM kernels.
#pragma once

#include "common.cuh"

namespace b200moe {

struct GemmArgs {
    const void* scale;
    const __nv_bfloat16* offset;
    const float* rowsum;  // [M] sum_k x[m,k]; only read when offset != nullptr
    const int64_t* group_list;
    __nv_bfloat16* y;
    int M, K, N, G, gl_type;
    int* status;
    // packed kernel only, optional: result row r goes to dst_base[row_code[r] >> 32] + (low 32 bits) * N
    // instead of y + r * N (rows handed back to the ranks they came from)
    const long long* row_code = nullptr;
    __nv_bfloat16* dst_base[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    int n_base = 0;
    long long dst_rows = 0;
    // int4 in one pass (grouped_gemm.cu), scratch of the call: the rows' exponents, the tiles that the two-pass kernel does again, and
    // [0] their number, [1] that kernel's ticket, [2] rows of x that are not exact in f16
    const int* row_exp = nullptr;
    int4* redo = nullptr;
    int* redo_ctl = nullptr;
};

// out[m] = sum_k x[m, k] in fp32 for the rows the group list uses, and status words 0 .. 3 zeroed (grouped_gemm.cu).
void launch_rowsum(const void* x, float* out, int64_t M, int64_t K, const int64_t* group_list, int64_t G, int gl_type,
                   int* status, cudaStream_t stream);

}  // namespace b200moe
