// Stand-alone per-token ops of the builtin surface (rms_norm, rope, sigmoid,
// mul, add, softmax, embedding) and the C-ABI entry points of the linear
// family.  The TL scripts call these builtins one by one
// (debug/chat_demo_with_kvcache.tl:219-290); the fused entry points in
// tlc_gemv.cu fold them into the GEMV launches.
#include <cmath>
#include <vector>

#include "tlc_gemm_wt.h"
#include "tlc_internal.h"

namespace {

// rms_norm_f16 (shaders/unified.metal:1785-1831) / Tensor::rms_norm_cpu
// (src/ops/normalization.rs:199-248): one CTA per row.  A launch of a few rows is a chain of latencies: the row is
// read once, a thread keeps its pieces, and the weights come with it, or before it where the caller vouches
// that no kernel in flight writes them (w_early): 32 x 4096 3.4 -> 2.3 us.
__global__ void __launch_bounds__(256) rms_norm_kernel(const __half *x, const __half *w,
                                                       __half *__restrict__ y, int d, float eps, int w_early) {
    constexpr int KEEP = 4;  // 16-byte pieces of the row a thread keeps: d = 8192
    __shared__ float warp_sums[8];
    const int tid = threadIdx.x, pieces = d >> 3;
    const __half *xr = x + (size_t)blockIdx.x * d;
    __half *yr = y + (size_t)blockIdx.x * d;
    // 16-byte accesses when the row allows it (d a multiple of 8, 16-byte aligned pointers)
    const bool vec = (d & 7) == 0 && ((((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) & 15) == 0);
    uint4 xv[KEEP], wv[KEEP];
    auto load = [&](const __half *src, uint4 (&v)[KEEP]) {
#pragma unroll
        for (int r = 0; r < KEEP; r++) {
            const int i = tid + r * 256;
            v[r] = i < pieces ? reinterpret_cast<const uint4 *>(src)[i] : make_uint4(0, 0, 0, 0);
        }
    };
    if (vec && w_early) load(w, wv);
    tlc_pdl_after_wait();
    float sq = 0.f;
    auto add = [&](const uint4 &raw) {
        const __half2 *h = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 v = __half22float2(h[j]);
            sq = fmaf(v.x, v.x, sq);
            sq = fmaf(v.y, v.y, sq);
        }
    };
    if (vec) {
        load(xr, xv);
        if (!w_early) load(w, wv);
#pragma unroll
        for (int r = 0; r < KEEP; r++) add(xv[r]);
        for (int i = tid + KEEP * 256; i < pieces; i += 256) add(reinterpret_cast<const uint4 *>(xr)[i]);
    } else {
        for (int i = tid; i < d; i += 256) {
            const float v = __half2float(xr[i]);
            sq = fmaf(v, v, sq);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((tid & 31) == 0) warp_sums[tid >> 5] = sq;
    __syncthreads();
    // (in the order of a shuffle tree over the eight sums)
    const float *s = warp_sums;
    const float total = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
    const float inv = 1.0f / sqrtf(total / (float)d + eps);
    auto store = [&](int i, const uint4 &raw, const uint4 &wraw) {
        const __half *xh = reinterpret_cast<const __half *>(&raw), *wh = reinterpret_cast<const __half *>(&wraw);
        __align__(16) __half o[8];
#pragma unroll
        for (int j = 0; j < 8; j++)
            o[j] = __float2half_rn(__fmul_rn(__fmul_rn(__half2float(xh[j]), inv), __half2float(wh[j])));
        reinterpret_cast<uint4 *>(yr)[i] = *reinterpret_cast<const uint4 *>(o);
    };
    if (vec) {
#pragma unroll
        for (int r = 0; r < KEEP; r++)
            if (tid + r * 256 < pieces) store(tid + r * 256, xv[r], wv[r]);
        for (int i = tid + KEEP * 256; i < pieces; i += 256)
            store(i, reinterpret_cast<const uint4 *>(xr)[i], reinterpret_cast<const uint4 *>(w)[i]);
    } else {
        for (int i = tid; i < d; i += 256) {
            const float nrm = __fmul_rn(__half2float(xr[i]), inv);
            yr[i] = __float2half_rn(__fmul_rn(nrm, __half2float(w[i])));
        }
    }
}

// rope_f16 (shaders/unified.metal:2355-2417): one thread per pair.
__global__ void rope_kernel(const __half *x, __half *__restrict__ y, int seq, int heads, int d,
                            int pos_offset, float base, const int *positions) {
    tlc_pdl_after_wait();
    const int half_d = d >> 1;
    const size_t total = (size_t)seq * heads * half_d;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int pair = (int)(i % half_d);
    const size_t sh = i / half_d;
    const int s = (int)(sh / heads);
    const unsigned pos = positions ? (unsigned)positions[s] : (unsigned)(s + pos_offset);
    const float exponent = (float)(2 * pair) / (float)d;
    const float freq = 1.0f / powf(base, exponent);
    const float theta = (float)pos * freq;
    const float cs = cosf(theta), sn = sinf(theta);
    const size_t o = sh * d + 2 * pair;
    const float x0 = __half2float(x[o]), x1 = __half2float(x[o + 1]);
    y[o] = __float2half_rn(__fsub_rn(__fmul_rn(x0, cs), __fmul_rn(x1, sn)));
    y[o + 1] = __float2half_rn(__fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, cs)));
}

// rope_candle_f16 (shaders/unified.metal:5122-5184): the same interleaved rotation with the
// cosines and sines read from f16 tables instead of being worked out.  Pair p of position s
// reads table[s * pitch + p] -- exactly the shader's index arithmetic (`seq_idx * head_dim +
// dim_pair_idx`, i.e. pitch = head_dim there).  One thread per pair.
__global__ void rope_table_kernel(const __half *x, const __half *cos_t,
                                  const __half *sin_t, __half *__restrict__ y, int seq, int heads, int d,
                                  int pitch) {
    tlc_pdl_after_wait();
    const int half_d = d >> 1;
    const size_t total = (size_t)seq * heads * half_d;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int pair = (int)(i % half_d);
    const size_t sh = i / half_d;
    const int s = (int)(sh / heads);
    const float cs = __half2float(cos_t[(size_t)s * pitch + pair]), sn = __half2float(sin_t[(size_t)s * pitch + pair]);
    const size_t o = sh * d + 2 * pair;
    const float x0 = __half2float(x[o]), x1 = __half2float(x[o + 1]);
    y[o] = __float2half_rn(__fsub_rn(__fmul_rn(x0, cs), __fmul_rn(x1, sn)));
    y[o + 1] = __float2half_rn(__fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, cs)));
}

// sigmoid: f32 math, RNE to f16 (Tensor::sigmoid_cpu, src/ops/activations.rs:252-266).
// One operation per element; eight elements a thread (16-byte accesses) where alignment allows.
struct OpSigmoid {
    static __device__ __forceinline__ __half run(__half x, __half) { return __float2half_rn(1.0f / (1.0f + expf(-__half2float(x)))); }
};
struct OpMul {
    static __device__ __forceinline__ __half run(__half a, __half b) { return __hmul(a, b); }
};
struct OpAdd {
    static __device__ __forceinline__ __half run(__half a, __half b) { return __hadd(a, b); }
};
struct OpSwiglu {  // silu(g) * u with the three f16 roundings of sigmoid, mul, mul
    static __device__ __forceinline__ __half run(__half g, __half u) { return __hmul(__hmul(g, OpSigmoid::run(g, g)), u); }
};
template <class OP, bool TWO>
__global__ void __launch_bounds__(256) elementwise_kernel(const __half *a, const __half *b,
                                                          __half *__restrict__ y, size_t n, int vec) {
    tlc_pdl_after_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (!vec) {
        if (i < n) y[i] = OP::run(a[i], TWO ? b[i] : a[i]);
        return;
    }
    if (i * 8 >= n) return;
    const uint4 av = reinterpret_cast<const uint4 *>(a)[i], bv = TWO ? reinterpret_cast<const uint4 *>(b)[i] : av;
    const __half *ah = reinterpret_cast<const __half *>(&av), *bh = reinterpret_cast<const __half *>(&bv);
    __align__(16) __half o[8];
#pragma unroll
    for (int j = 0; j < 8; j++) o[j] = OP::run(ah[j], bh[j]);
    reinterpret_cast<uint4 *>(y)[i] = *reinterpret_cast<const uint4 *>(o);
}
// softmax over the last dim, one warp per row; arithmetic of
// softmax_simple_f16 (shaders/unified.metal:2150-2200): finite-only f32 max and
// sum, exponentials rounded to f16 before the divide, uniform row when the sum
// degenerates.
__global__ void softmax_kernel(const __half *x, __half *__restrict__ y, int rows, int last) {
    tlc_pdl_after_wait();
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const __half *xr = x + (size_t)row * last;
    __half *yr = y + (size_t)row * last;
    float mx = -INFINITY;
    for (int i = lane; i < last; i += 32) {
        float v = __half2float(xr[i]);
        if (isfinite(v)) mx = fmaxf(mx, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (!isfinite(mx)) mx = 0.f;
    float sum = 0.f;
    for (int i = lane; i < last; i += 32) {
        float v = __half2float(xr[i]);
        sum += isfinite(v) ? expf(v - mx) : 0.f;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (sum > 0.f && isfinite(sum)) {
        for (int i = lane; i < last; i += 32) {
            float v = __half2float(xr[i]);
            float e = isfinite(v) ? expf(v - mx) : 0.f;
            yr[i] = __float2half_rn(__half2float(__float2half_rn(e)) / sum);
        }
    } else {
        const __half u = __float2half_rn(1.0f / (float)last);
        for (int i = lane; i < last; i += 32) yr[i] = u;
    }
}

// embedding_lookup_f16 (shaders/unified.metal:658-675): 16-byte vector gather.
__global__ void embedding_kernel(const __half *table, const int *ids, int d,
                                 int m, __half *__restrict__ y) {
    tlc_pdl_after_wait();
    const int vec_per_row = d >> 3;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)m * vec_per_row) return;
    const int r = (int)(i / vec_per_row), c = (int)(i % vec_per_row);
    reinterpret_cast<uint4 *>(y + (size_t)r * d)[c] =
        reinterpret_cast<const uint4 *>(table + (size_t)ids[r] * d)[c];
}
__global__ void embedding_scalar_kernel(const __half *table, const int *ids, int d,
                                        int m, __half *__restrict__ y) {
    tlc_pdl_after_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)m * d) return;
    const int r = (int)(i / d), c = (int)(i % d);
    y[i] = table[(size_t)ids[r] * d + c];
}

// Launch on the context's stream with programmatic dependent launch.
template <typename... KArgs, typename... Args>
int32_t launch_op(tlc_ctx *ctx, void (*kernel)(KArgs...), unsigned grid, unsigned block, Args &&...args) {
    const cudaError_t le = tlc_launch_pdl(ctx, kernel, dim3(grid), dim3(block), 0, args...);
    if (le != cudaSuccess) {
        cudaGetLastError();
        return tlc_fail(TLC_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(le));
    }
    TLC_CHECK_LAUNCH(ctx);
    return TLC_OK;
}

inline unsigned blocks_for(size_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

int32_t tlc_launch_rms_norm(tlc_ctx *ctx, const void *x_dev, const void *w_dev, void *y_dev, int32_t rows, int32_t d, float eps,
                            bool w_early) {
    return launch_op(ctx, rms_norm_kernel, rows, 256, static_cast<const __half *>(x_dev), static_cast<const __half *>(w_dev),
                     static_cast<__half *>(y_dev), d, eps, w_early ? 1 : 0);
}

extern "C" int32_t tlc_rms_norm(tlc_ctx *ctx, const void *x_dev, const void *w_dev, void *y_dev, int32_t rows,
                                int32_t d, float eps) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    tlc_perf_scope perf(ctx, "rms_norm(rows=%d, d=%d)", rows, d);
    TLC_REQUIRE(x_dev && w_dev && y_dev, TLC_ERR_INVALID_OPERATION, "rms_norm: null pointer");
    TLC_REQUIRE(rows >= 0 && d > 0, TLC_ERR_INVALID_DIMENSION, "rms_norm: bad shape [%d, %d]", rows, d);
    if (rows == 0) return TLC_OK;
    return tlc_launch_rms_norm(ctx, x_dev, w_dev, y_dev, rows, d, eps, false);
}

extern "C" int32_t tlc_rope(tlc_ctx *ctx, const void *x_dev, void *y_dev, int32_t seq, int32_t heads,
                            int32_t d, int32_t pos_offset, uint32_t base, const int32_t *positions_dev) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    tlc_perf_scope perf(ctx, "rope(seq=%d, heads=%d, d=%d)", seq, heads, d);
    TLC_REQUIRE(x_dev && y_dev, TLC_ERR_INVALID_OPERATION, "rope: null pointer");
    // Tensor::rope rejects an odd head_dim (src/ops/rope.rs:90-96).
    TLC_REQUIRE(d > 0 && d % 2 == 0, TLC_ERR_INVALID_OPERATION, "RoPE requires even head_dim, got %d", d);
    TLC_REQUIRE(seq >= 0 && heads > 0, TLC_ERR_INVALID_DIMENSION, "rope: bad shape [%d, %d, %d]", seq, heads, d);
    if (seq == 0) return TLC_OK;
    const size_t total = (size_t)seq * heads * (d / 2);
    return launch_op(ctx, rope_kernel, blocks_for(total, 256), 256, 
        static_cast<const __half *>(x_dev), static_cast<__half *>(y_dev), seq, heads, d, pos_offset, (float)base,
        positions_dev);
}

// rope(x, cos, sin): the arm of the rope builtin that takes precomputed tables
// (src/interpreter/builtin_tensor.rs:634-722 -> Tensor::rope_candle, src/ops/rope.rs:18-65).
// x, y: [seq, heads, d] f16; cos/sin: f16 tables of table_rows rows, `pitch` elements apart;
// pair p of position s uses cos[s * pitch + p], sin[s * pitch + p].
//   * A table of head_dim / 2 columns (pitch = head_dim / 2, one column per rotary pair) is what
//     the kernel's index arithmetic is written for, and gives the same rotation as tlc_rope.
//   * The reference's own builtin stores every frequency twice in rows of head_dim values and
//     passes pitch = head_dim in effect: pair p then reads column p of a row laid out
//     c0 c0 c1 c1 ..., i.e. frequency p / 2 -- its result, quirk included, is reproduced by
//     passing that table with pitch = head_dim.
extern "C" int32_t tlc_rope_table(tlc_ctx *ctx, const void *x_dev, const void *cos_dev, const void *sin_dev,
                                  void *y_dev, int32_t seq, int32_t heads, int32_t d, int32_t table_rows,
                                  int32_t pitch) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    tlc_perf_scope perf(ctx, "rope_table(seq=%d, heads=%d, d=%d)", seq, heads, d);
    TLC_REQUIRE(x_dev && cos_dev && sin_dev && y_dev, TLC_ERR_INVALID_OPERATION, "rope: null pointer");
    TLC_REQUIRE(d > 0 && d % 2 == 0, TLC_ERR_INVALID_OPERATION, "RoPE requires even head_dim, got %d", d);
    TLC_REQUIRE(seq >= 0 && heads > 0, TLC_ERR_INVALID_DIMENSION, "rope: bad shape [%d, %d, %d]", seq, heads, d);
    TLC_REQUIRE(pitch >= d / 2, TLC_ERR_INVALID_OPERATION,
                "cos/sin last dim must hold head_dim / 2 = %d pairs, got %d", d / 2, pitch);
    TLC_REQUIRE(table_rows >= seq, TLC_ERR_INVALID_OPERATION,
                "cos/sin first dim must be >= seq_len = %d, got cos: %d, sin: %d", seq, table_rows, table_rows);
    if (seq == 0) return TLC_OK;
    const size_t total = (size_t)seq * heads * (d / 2);
    return launch_op(ctx, rope_table_kernel, blocks_for(total, 256), 256, 
        static_cast<const __half *>(x_dev), static_cast<const __half *>(cos_dev), static_cast<const __half *>(sin_dev),
        static_cast<__half *>(y_dev), seq, heads, d, pitch);
}

// matmul(a, b): a [m, k] . b [k2, n] -> y [m, n], all f16 on the device.  Shape rule and message
// of Tensor::matmul (src/ops/matmul.rs:36-46).
extern "C" int32_t tlc_matmul(tlc_ctx *ctx, const void *a_dev, const void *b_dev, void *y_dev, int32_t m, int32_t k,
                              int32_t k2, int32_t n) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    tlc_perf_scope perf(ctx, "matmul(m=%d, k=%d, n=%d)", m, k, n);
    TLC_REQUIRE(a_dev && b_dev && y_dev, TLC_ERR_INVALID_OPERATION, "matmul: null pointer");
    TLC_REQUIRE(m >= 0 && k >= 0 && k2 >= 0 && n >= 0, TLC_ERR_INVALID_DIMENSION, "matmul: bad shape");
    TLC_REQUIRE(k == k2, TLC_ERR_INVALID_OPERATION, "matmul shape mismatch: [%d, %d] @ [%d, %d]", m, k, k2, n);
    if (m == 0 || n == 0) return TLC_OK;
    if (k > 0) return tlc_launch_matmul_f16(ctx, a_dev, b_dev, y_dev, m, k, n);
    TLC_CUDA(cudaMemsetAsync(y_dev, 0, (size_t)m * n * 2, ctx->stream));  // a sum of nothing
    return TLC_OK;
}

template <class OP, bool TWO>
static int32_t elementwise(tlc_ctx *ctx, const char *name, const void *a, const void *b, void *y, size_t n) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    TLC_REQUIRE(a && (b || !TWO) && y, TLC_ERR_INVALID_OPERATION, "tlc_%s: null pointer", name);
    if (n == 0) return TLC_OK;
    tlc_perf_scope perf(ctx, "%s(n=%zu)", name, n);
    const int vec = n % 8 == 0 && (((uintptr_t)a | (uintptr_t)(TWO ? b : nullptr) | (uintptr_t)y) & 15) == 0 ? 1 : 0;
    return launch_op(ctx, elementwise_kernel<OP, TWO>, blocks_for(vec ? n / 8 : n, 256), 256, static_cast<const __half *>(a),
                     static_cast<const __half *>(b), static_cast<__half *>(y), n, vec);
}
extern "C" int32_t tlc_sigmoid(tlc_ctx *ctx, const void *x_dev, void *y_dev, size_t n) {
    return elementwise<OpSigmoid, false>(ctx, "sigmoid", x_dev, nullptr, y_dev, n);
}
extern "C" int32_t tlc_mul(tlc_ctx *ctx, const void *a_dev, const void *b_dev, void *y_dev, size_t n) {
    return elementwise<OpMul, true>(ctx, "mul", a_dev, b_dev, y_dev, n);
}
extern "C" int32_t tlc_add(tlc_ctx *ctx, const void *a_dev, const void *b_dev, void *y_dev, size_t n) {
    return elementwise<OpAdd, true>(ctx, "add", a_dev, b_dev, y_dev, n);
}
extern "C" int32_t tlc_swiglu(tlc_ctx *ctx, const void *a_dev, const void *b_dev, void *y_dev, size_t n) {
    return elementwise<OpSwiglu, true>(ctx, "swiglu", a_dev, b_dev, y_dev, n);
}

extern "C" int32_t tlc_softmax(tlc_ctx *ctx, const void *x_dev, void *y_dev, int32_t rows, int32_t last_dim) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    tlc_perf_scope perf(ctx, "softmax(rows=%d, d=%d)", rows, last_dim);
    TLC_REQUIRE(x_dev && y_dev, TLC_ERR_INVALID_OPERATION, "softmax: null pointer");
    TLC_REQUIRE(rows >= 0 && last_dim > 0, TLC_ERR_INVALID_DIMENSION, "softmax: bad shape [%d, %d]", rows, last_dim);
    if (rows == 0) return TLC_OK;
    return launch_op(ctx, softmax_kernel, blocks_for((size_t)rows * 32, 256), 256, 
        static_cast<const __half *>(x_dev), static_cast<__half *>(y_dev), rows, last_dim);
}

extern "C" int32_t tlc_embedding(tlc_ctx *ctx, const void *table_dev, int32_t vocab, int32_t d,
                                 const int32_t *ids_host, int32_t m, void *y_dev) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    tlc_perf_scope perf(ctx, "embedding(d=%d)", d);
    TLC_REQUIRE(table_dev && ids_host && y_dev, TLC_ERR_INVALID_OPERATION, "embedding: null pointer");
    TLC_REQUIRE(vocab > 0 && d > 0 && m >= 0, TLC_ERR_INVALID_DIMENSION, "embedding: bad shape");
    // Host-side bounds check as in src/interpreter/builtin_nn.rs:681-688.
    for (int i = 0; i < m; i++)
        TLC_REQUIRE(ids_host[i] >= 0 && ids_host[i] < vocab, TLC_ERR_INDEX,
                    "Index out of bounds: index %d, size %d", ids_host[i], vocab);
    if (m == 0) return TLC_OK;
    tlc_buf *ids = nullptr;
    if (int32_t rc = tlc_alloc(ctx, (size_t)m * sizeof(int32_t), &ids)) return rc;
    cudaError_t e = cudaMemcpyAsync(ids->ptr, ids_host, (size_t)m * sizeof(int32_t), cudaMemcpyHostToDevice,
                                    ctx->stream);
    if (e != cudaSuccess) {
        tlc_free(ids);
        return tlc_fail(TLC_ERR_CUDA, "embedding: id upload failed: %s", cudaGetErrorString(e));
    }
    const bool vec = d % 8 == 0 && ((uintptr_t)table_dev % 16 == 0) && ((uintptr_t)y_dev % 16 == 0);
    int32_t rc;
    if (vec)
        rc = launch_op(ctx, embedding_kernel, blocks_for((size_t)m * (d / 8), 256), 256, 
            static_cast<const __half *>(table_dev), static_cast<const int *>(ids->ptr), d, m,
            static_cast<__half *>(y_dev));
    else
        rc = launch_op(ctx, embedding_scalar_kernel, blocks_for((size_t)m * d, 256), 256, 
            static_cast<const __half *>(table_dev), static_cast<const int *>(ids->ptr), d, m,
            static_cast<__half *>(y_dev));
    tlc_free(ids);  // stream-ordered: the gather above is already queued
    return rc;
}

// ---- linear family -----------------------------------------------------------

static int32_t check_linear(tlc_ctx *ctx, tlc_qtensor *w, const void *x, int32_t m, int64_t x_cols,
                            const void *y) {
    TLC_REQUIRE(w && x && y, TLC_ERR_INVALID_OPERATION, "linear: null pointer");
    TLC_REQUIRE(m >= 1, TLC_ERR_INVALID_OPERATION, "matmul_transposed_b requires 2D tensors (m = %d)", m);
    // Same message shape as src/ops/matmul.rs:266-273.
    TLC_REQUIRE(x_cols == w->n_cols, TLC_ERR_INVALID_OPERATION,
                "matmul_transposed_b shape mismatch: [%d, %lld] @ [%lld, %lld].T", m, (long long)x_cols,
                (long long)w->n_rows, (long long)w->n_cols);
    TLC_REQUIRE(w->ctx->device == ctx->device, TLC_ERR_DEVICE,
                "matmul_transposed_b requires tensors on same device");
    return TLC_OK;
}

static const char *type_name(const tlc_qtensor *w) {
    return !w ? "?" : w->type == TLC_TYPE_Q4_0 ? "q4_0" : w->type == TLC_TYPE_Q8_0 ? "q8_0" : w->type == TLC_TYPE_Q6_K ? "q6_k" : "f16";
}

extern "C" int32_t tlc_linear(tlc_ctx *ctx, tlc_qtensor *w, const void *x_dev, int32_t m, int64_t x_cols,
                              void *y_dev, const void *bias_dev) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    if (int32_t rc = check_linear(ctx, w, x_dev, m, x_cols, y_dev)) return rc;
    tlc_perf_scope perf(ctx, "linear(%s, m=%d, n=%lld, k=%lld)", type_name(w), m, (long long)w->n_rows, (long long)w->n_cols);
    tlc_gemv_args a;
    a.n_out = 1;
    a.outs[0] = {w, y_dev, 0};
    a.x = x_dev;
    a.m = m;
    a.bias = bias_dev;
    return tlc_launch_gemv(ctx, a);
}

extern "C" int32_t tlc_linear_host(tlc_ctx *ctx, tlc_qtensor *w, const void *x_host, int32_t m,
                                   int64_t x_cols, void *y_host, const void *bias_host) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    if (int32_t rc = check_linear(ctx, w, x_host, m, x_cols, y_host)) return rc;
    const size_t xb = (size_t)m * x_cols * 2, yb = (size_t)m * w->n_rows * 2, bb = (size_t)w->n_rows * 2;
    tlc_buf *xd = nullptr, *yd = nullptr, *bd = nullptr;
    int32_t rc = tlc_alloc(ctx, xb, &xd);
    if (!rc) rc = tlc_alloc(ctx, yb, &yd);
    if (!rc && bias_host) rc = tlc_alloc(ctx, bb, &bd);
    if (!rc) rc = tlc_upload(ctx, xd->ptr, x_host, xb);
    if (!rc && bias_host) rc = tlc_upload(ctx, bd->ptr, bias_host, bb);
    if (!rc) rc = tlc_linear(ctx, w, xd->ptr, m, x_cols, yd->ptr, bd ? bd->ptr : nullptr);
    if (!rc) rc = tlc_download(ctx, y_host, yd->ptr, yb);
    tlc_free(xd);
    tlc_free(yd);
    tlc_free(bd);
    return rc;
}

extern "C" int32_t tlc_norm_linear_multi(tlc_ctx *ctx, int32_t n_weights, tlc_qtensor *const *w,
                                         void *const *y_dev, const int32_t *rope_heads, const void *x_dev,
                                         int32_t m, const void *norm_w_dev, float eps, int32_t pos_offset,
                                         uint32_t rope_base, const int32_t *positions_dev) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    TLC_REQUIRE(n_weights >= 1 && n_weights <= 3 && w && y_dev, TLC_ERR_INVALID_OPERATION,
                "norm_linear_multi: 1..3 weights expected, got %d", n_weights);
    tlc_gemv_args a;
    a.n_out = n_weights;
    for (int i = 0; i < n_weights; i++) {
        if (int32_t rc = check_linear(ctx, w[i], x_dev, m, w[0] ? w[0]->n_cols : 0, y_dev[i])) return rc;
        a.outs[i] = {w[i], y_dev[i], rope_heads ? rope_heads[i] : 0};
    }
    a.x = x_dev;
    a.m = m;
    a.norm_w = norm_w_dev;
    a.eps = eps;
    a.pos_offset = pos_offset;
    a.rope_base = rope_base;
    a.positions = positions_dev;
    tlc_perf_scope perf(ctx, "norm_linear_multi(%s, %d weights, m=%d, k=%lld)", type_name(w[0]), n_weights, m,
                        (long long)w[0]->n_cols);
    return tlc_launch_gemv(ctx, a);
}

extern "C" int32_t tlc_swiglu_gate_up(tlc_ctx *ctx, tlc_qtensor *w_gate, tlc_qtensor *w_up, const void *x_dev,
                                      int32_t m, const void *norm_w_dev, float eps, void *act_dev) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    if (int32_t rc = check_linear(ctx, w_gate, x_dev, m, w_gate ? w_gate->n_cols : 0, act_dev)) return rc;
    if (int32_t rc = check_linear(ctx, w_up, x_dev, m, w_gate->n_cols, act_dev)) return rc;
    tlc_gemv_args a;
    a.n_out = 2;
    a.outs[0] = {w_gate, act_dev, 0};
    a.outs[1] = {w_up, act_dev, 0};
    a.x = x_dev;
    a.m = m;
    a.norm_w = norm_w_dev;
    a.eps = eps;
    a.epilogue = TLC_EPI_SWIGLU;
    tlc_perf_scope perf(ctx, "swiglu_gate_up(%s, m=%d, n=%lld, k=%lld)", type_name(w_gate), m, (long long)w_gate->n_rows,
                        (long long)w_gate->n_cols);
    return tlc_launch_gemv(ctx, a);
}

extern "C" int32_t tlc_linear_residual(tlc_ctx *ctx, tlc_qtensor *w, const void *x_dev, int32_t m,
                                       const void *residual_dev, void *y_dev) {
    if (int32_t rc = tlc_enter(ctx)) return rc;
    if (int32_t rc = check_linear(ctx, w, x_dev, m, w ? w->n_cols : 0, y_dev)) return rc;
    TLC_REQUIRE(residual_dev, TLC_ERR_INVALID_OPERATION, "linear_residual: null residual");
    tlc_gemv_args a;
    a.n_out = 1;
    a.outs[0] = {w, y_dev, 0};
    a.x = x_dev;
    a.m = m;
    a.epilogue = TLC_EPI_RESIDUAL;
    a.residual = residual_dev;
    tlc_perf_scope perf(ctx, "linear_residual(%s, m=%d, n=%lld, k=%lld)", type_name(w), m, (long long)w->n_rows,
                        (long long)w->n_cols);
    return tlc_launch_gemv(ctx, a);
}
