// bf16 products of at most GR_MAX_ROWS rows (gemm_rows_sm100.cu); operands checked by the caller (gemm_bf16_sm100.cu).
#pragma once

#include "common.cuh"

namespace bn {

constexpr int GR_MAX_ROWS = 128;

struct RowsGemm {
    const void *a, *w;             // (M, K), and (N, K): the output's columns, or (glu) their gate and up rows 128 by 128
    __nv_bfloat16* c;              // (M, n_out), or
    float* c32;                    // the sums themselves
    const __nv_bfloat16* mul;      // optional: c = act(sum) * mul, (M, mul_ld)
    const float* bias;             // optional: c = act(sum + bias)
    int* error_word;
    long long mul_ld;
    int M, N, K, n_out, act;
    bool glu;
};

// whether gemm_rows is the kernel for a product of M rows with n_out columns (glu: of gate and up each)
bool gemm_rows_ok(int M, int n_out, int K, bool glu);
int gemm_rows(const RowsGemm& p, cudaStream_t st, const char* what);

}  // namespace bn
