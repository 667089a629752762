// Matrix products with the weight rows on the M side of the MMA (tlc_gemm_wt.cu).
#pragma once

#include "tlc_internal.h"

namespace tlc_gemm {

// What the A operand is made from: Q4_0 / Q8_0 tiles, f16 rows along K, or a dense [K, N] matrix.
enum WtSource { kWtQ4 = 2, kWtQ8 = 8, kWtF16 = 1, kWtF16T = 101 };

}  // namespace tlc_gemm

// The contract of tlc_launch_gemv for Q4_0 / Q8_0 weights; norm_w is not handled here (a.x is what is multiplied).
int32_t tlc_launch_gemm_wt(tlc_ctx *ctx, const tlc_gemv_args &a);
// y[m, n] = x[m, k] . W^T (w [n, k], rows w_pitch bytes apart) + bias / residual, dense f16.
int32_t tlc_launch_gemm_f16(tlc_ctx *ctx, const void *w, size_t w_pitch, int n, int k, const void *x, int m, void *y,
                            const void *bias, const void *residual);
// c[m, n] = a[m, k] . b[k, n], dense f16.
int32_t tlc_launch_matmul_f16(tlc_ctx *ctx, const void *a, const void *b, void *c, int m, int k, int n);
