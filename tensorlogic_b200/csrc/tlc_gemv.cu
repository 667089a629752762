// Fused dequant-GEMV for decode-sized activations (M <= 16) over weights kept
// as GGUF Q4_0 / Q8_0 blocks in 16-row tiles (tlc_tile.cuh).
//
// Takes the place of the dense f16 kernels the reference runs after
// dequantizing at load time (matmul_transposed_b_tiled_f16,
// shaders/unified.metal:4226-4347, dispatched from src/ops/matmul.rs:314-458)
// and of the separate rms_norm / rope / sigmoid / mul / add launches around
// them in the TL scripts (debug/chat_demo_with_kvcache.tl:219-290).
//
// Common to both kernels (the weight bytes are read from HBM exactly once):
//   * persistent CTAs, up to two per SM, each walking 16-row slabs of the weight(s); the tiles of a slab
//     arrive through a shared memory ring in bulk async copies (a slab's tiles are contiguous in HBM),
//     completing on mbarriers -- no thread ever issues a narrow global load for weight data, and the
//     ring keeps tens of KB per SM in flight independent of occupancy;
//   * consumer warps read their fragment words with two conflict-free 16-byte shared loads per tile and
//     unpack nibbles / bytes in registers straight into f16 tensor-core fragments: a 4-bit (8-bit) integer n
//     placed in the low mantissa bits of a binary16 is the subnormal n * 2^-24, so one AND per pair of
//     weights yields an exact A fragment; the -8 (-128) offset is carried by the accumulator's initial value
//     (-8 * sum of the 32 activations of the block) and the block scale d multiplies the 16x8 block
//     result in f32;  mma.sync m16n8k16 with f32 accumulation does the dot products for up to 8
//     activation rows at no extra cost (8 clocks per sub-core, as long as the unpacking of its block takes
//     the integer pipe, which needs two clocks an operation);
//   * the K range of a slab is split over the warps, reduced through shared memory (several slabs per
//     reduction), and the epilogue (f16 rounding, bias / residual add, SiLU(gate)*up, interleaved RoPE)
//     is applied before the single store.
// One row (tlc_gemv_row1.cuh): the row, optionally RMS-normalised, lies in shared memory in fragment order.
// 2 to 16 rows (tlc_gemv_kernel.cuh): that copy would be read 512 bytes a block and warp, by far more than the
// weights, and crowd out the ring.  Each warp keeps its share of K of all rows in registers for the whole
// launch instead, a K longer than a CTA's registers hold is shared out over a thread-block cluster,
// and the RMSNorm is done once by a kernel of its own (frag_rows_kernel) and not by every CTA.  Measured on one
// B200, before -> now: Q4_0 4096 x 4096, 8 rows 10.1 -> 7.4 us; norm + 7168 x 8192 at 8 / 16 rows 31.2 -> 16.8 /
// 43.8 -> 21.9 us; norm + 2560 x 2048 at 5 / 16 rows 9.5 -> 6.9 / 19.3 -> 8.2 us; 28672 x 8192 at 8 rows 42.8 -> 33.2 us.
#include <cuda_fp16.h>

#include <cstring>

#include "tlc_gemm_kernel.cuh"
#include "tlc_gemm_wt.h"
#include "tlc_gemv_kernel.cuh"
#include "tlc_gemv_row1.cuh"
#include "tlc_internal.h"
#include "tlc_tile.cuh"

using namespace tlc_gemv;

namespace {

// ---------------------------------------------------------------------------
// Generic path for dense f16 weights: any M, no alignment assumptions.  One
// warp per output row -- correct but far from the roofline.
// ---------------------------------------------------------------------------
__global__ void linear_generic_kernel(const uint8_t *__restrict__ w, size_t pitch, int n_rows, int k, const __half *__restrict__ x, int m, __half *__restrict__ y,
                                      const __half *__restrict__ bias) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= n_rows) return;
    const __half *wr = reinterpret_cast<const __half *>(w + (size_t)warp * pitch);
    for (int mm = 0; mm < m; mm++) {
        const __half *xr = x + (size_t)mm * k;
        float acc = 0.f;
        for (int i = lane; i < k; i += 32) acc = fmaf(__half2float(wr[i]), __half2float(xr[i]), acc);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) {
            __half h = __float2half_rn(acc);
            if (bias) h = __hadd(h, bias[warp]);
            y[(size_t)mm * n_rows + warp] = h;
        }
    }
}

// ---------------------------------------------------------------------------
// Dense f16 weights (F16 / F32 files, Q6_K after its load-time dequantization,
// tied embeddings), one activation row: one warp per output row, 16-byte loads of the row and of
// the activations, f32 accumulation, optional bias / residual.  HBM-bound on the 2 bytes
// per weight; K must be a multiple of 8 and rows 16-byte aligned.  (More rows: tlc_gemm_wt.cu.)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) linear_f16_kernel(const uint8_t *__restrict__ w, size_t pitch, int n_rows, int k,
                                                         const __half *x, __half *__restrict__ y, const __half *bias,
                                                         const __half *residual) {
    tlc_pdl_prologue();
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= n_rows) return;
    const uint4 *wr = reinterpret_cast<const uint4 *>(w + (size_t)row * pitch);
    const int steps = k >> 3;  // 16-byte pieces per row
    float acc = 0.f;
#pragma unroll 4
    for (int s = lane; s < steps; s += 32) {
        const uint4 wv = __ldg(wr + s), xv = *(reinterpret_cast<const uint4 *>(x) + s);
        const __half2 *wh = reinterpret_cast<const __half2 *>(&wv), *xh = reinterpret_cast<const __half2 *>(&xv);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 wf = __half22float2(wh[j]), xf = __half22float2(xh[j]);
            acc = fmaf(wf.x, xf.x, acc);
            acc = fmaf(wf.y, xf.y, acc);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
        __half h = __float2half_rn(acc);
        if (bias) h = __hadd(h, bias[row]);
        if (residual) h = __hadd(h, residual[row]);
        y[row] = h;
    }
}

// Q6_K rows of more than 65536 columns, whose activations a launch of the GEMV cannot hold: one warp per output row,
// any K and any number of activation rows, the arithmetic of the GEMV (integers times the group's scale, f32 sums).
__global__ void __launch_bounds__(256) linear_q6k_long_kernel(const uint8_t *__restrict__ w, size_t pitch, int n_rows, int k,
                                                              const __half *x, int m, __half *__restrict__ y, const __half *bias,
                                                              const __half *residual) {
    tlc_pdl_after_wait();
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= n_rows) return;
    for (int mm = 0; mm < m; mm++) {
        const __half *xr = x + (size_t)mm * k + lane;
        float acc = 0.f;
        for (int sb = 0; sb < k >> 8; sb++) {
            const uint8_t *blk = w + (size_t)row * pitch + (size_t)sb * 224;
            const float d = __half2float(*reinterpret_cast<const __half *>(blk + 208));
#pragma unroll
            for (int g = 0; g < 8; g++) {  // elements 32 g + lane: half h, quarter j of it
                const int h = g >> 2, j = g & 3;
                const int lo = blk[64 * h + 32 * (j & 1) + lane] >> (j >= 2 ? 4 : 0) & 15, hi = blk[128 + 32 * h + lane] >> (2 * j) & 3;
                const float scale = d * (float)reinterpret_cast<const int8_t *>(blk + 192)[8 * h + (lane >> 4) + 2 * j];
                acc = fmaf(scale, (float)((lo | hi << 4) - 32) * __half2float(xr[sb * 256 + 32 * g]), acc);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) {
            __half v = __float2half_rn(acc);
            if (bias) v = __hadd(v, bias[row]);
            if (residual) v = __hadd(v, residual[(size_t)mm * n_rows + row]);
            y[(size_t)mm * n_rows + row] = v;
        }
    }
}

// Launches a GEMV kernel (fn) in `threads`-wide CTAs with all the shared memory it asks for, PDL and, with
// p.ksplit > 1, clusters; `configured` belongs to fn.
int32_t launch_kernel(tlc_ctx *ctx, void (*fn)(GemvParams), bool (&configured)[64], const GemvParams &p, int grid, int threads,
                      size_t smem) {
    if (!configured[ctx->device & 63]) {
        TLC_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ctx->prop.sharedMemPerBlockOptin));
        TLC_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        TLC_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        configured[ctx->device & 63] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (ctx->use_pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.ksplit > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)p.ksplit;
        attr[na].val.clusterDim.y = 1;
        attr[na++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    cudaError_t le = cudaLaunchKernelEx(&cfg, fn, p);
    if (le != cudaSuccess) {
        cudaGetLastError();
        return tlc_fail(TLC_ERR_CUDA, "gemv launch failed: %s", cudaGetErrorString(le));
    }
    TLC_CHECK_LAUNCH(ctx);
    return TLC_OK;
}
template <int QT, int NT, int TI, int CW>
int32_t launch_rows(tlc_ctx *ctx, const GemvParams &p, int grid, size_t smem) {
    static bool configured[64] = {};
    return launch_kernel(ctx, gemv_mma_kernel<QT, NT, TI, CW>, configured, p, grid, CW * 32, smem);
}
template <int QT, int AS, int CW>
int32_t launch_row1_as(tlc_ctx *ctx, const GemvParams &p, int grid, size_t smem) {
    static bool configured[64] = {};
    return launch_kernel(ctx, gemv_row1_kernel<QT, AS, CW>, configured, p, grid, (CW + 1) * 32, smem);
}

// One activation row.
template <int QT>
int32_t launch_row1(tlc_ctx *ctx, GemvParams &p) {
    constexpr size_t STAGE_BYTES = (size_t)kTilesPerStage * QTraits<QT>::TILE_BYTES;
    p.ksplit = 1;
    p.nblk_pad = p.ktiles * QTraits<QT>::TB;
    p.nchunks = (p.ktiles + kTilesPerStage - 1) / kTilesPerStage;
    const size_t budget = (size_t)ctx->prop.sharedMemPerBlockOptin;
    TLC_REQUIRE(row1_fixed_smem(p.nblk_pad, p.subs) + 2 * STAGE_BYTES <= budget, TLC_ERR_INVALID_OPERATION,
                "gemv: K = %d too large for the shared-memory staging", p.k);
    // Two CTAs per SM (16 consumer warps hide the shared-memory and MMA latency
    // of the unpack loop) whenever the activations leave room for at least
    // three ring stages in half of the SM's shared memory.
    const size_t half = (size_t)ctx->prop.sharedMemPerMultiprocessor / 2 - 1024;
    // (Measured on the TinyLlama decode step: keeping small launches at one CTA per
    // SM, to leave room for the next kernel's early CTAs, costs 8 % against
    // letting them spread over two CTAs per SM.)
    const bool two = row1_fixed_smem(p.nblk_pad, p.subs) + 3 * STAGE_BYTES <= half;
    // One CTA per SM: sixteen consumer warps instead of eight, if three ring stages remain.
    const int cw = !two && row1_fixed_smem(p.nblk_pad, p.subs, 16) + 3 * STAGE_BYTES <= budget ? 16 : 8;
    const size_t cap = two ? half : budget;
    const int max_ctas = two ? 2 * ctx->sm_count : ctx->sm_count;
    const int grid = p.total_units < max_ctas ? p.total_units : max_ctas;
    // Accumulator sets per reduction: enough units for about four ring stages
    // between two cross-warp reductions, as far as this CTA has units.
    const int units_per_cta = (p.total_units + grid - 1) / grid;
    const int iters_per_unit = p.subs * p.nchunks;
    int ub = (4 + iters_per_unit - 1) / iters_per_unit;
    if (ub > units_per_cta) ub = units_per_cta;
    int as = p.subs;
    while (as < ub * p.subs && as < 4) as *= 2;
    const size_t smem_fixed = row1_fixed_smem(p.nblk_pad, as, cw);
    // No more stages than this CTA will ever fill.
    const long per_cta = (long)units_per_cta * p.subs * p.nchunks;
    int stages = (int)((cap - smem_fixed) / STAGE_BYTES);
    if (stages > kMaxStages) stages = kMaxStages;
    if (stages > per_cta) stages = per_cta < 2 ? 2 : (int)per_cta;
    p.nstages = stages;
    // Mode 4 decides per launch.  A kernel whose CTAs stream eight or more ring stages (40 MB over the
    // grid, about 6 us of HBM time) lets its successor in right after its own dependency wait: the
    // successor is then resident with its ring filled when this grid ends (Llama-70B decode: 10.07 ->
    // 9.74 ms per token).  Shorter kernels keep the late trigger (TinyLlama decode: 2.2 % slower with
    // the early one from three stages on, 0.5 % slower with it everywhere).
    p.pdl_mode = ctx->pdl_mode == 4 ? (per_cta >= 8 ? 3 : 2) : ctx->pdl_mode;
    p.contig = units_per_cta <= 4 ? 1 : 0;
    const size_t smem = smem_fixed + (size_t)stages * STAGE_BYTES;
    if (cw == 16)
        return as == 1   ? launch_row1_as<QT, 1, 16>(ctx, p, grid, smem)
               : as == 2 ? launch_row1_as<QT, 2, 16>(ctx, p, grid, smem)
                         : launch_row1_as<QT, 4, 16>(ctx, p, grid, smem);
    return as == 1   ? launch_row1_as<QT, 1, 8>(ctx, p, grid, smem)
           : as == 2 ? launch_row1_as<QT, 2, 8>(ctx, p, grid, smem)
                     : launch_row1_as<QT, 4, 8>(ctx, p, grid, smem);
}

// Clusters of ks sixteen-warp CTAs that the device holds at once (asked once, with all of the shared memory).
int gemv_clusters(tlc_ctx *ctx, int ks) {
    static int known[64][17];
    int &n = known[ctx->device & 63][ks];
    if (n == 0) {
        auto fn = gemv_mma_kernel<TLC_TYPE_Q4_0, 1, 1, 16>;
        cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ctx->prop.sharedMemPerBlockOptin);
        cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)ks);
        cfg.blockDim = dim3(16 * 32);
        cfg.dynamicSmemBytes = ctx->prop.sharedMemPerBlockOptin - 2048;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)ks;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = -1;
        }
    }
    return n;
}

// Tiles along K that one launch can hold the activations of, per row tile count.
constexpr int kMaxCluster = 16;
template <int QT> constexpr int max_window(int nt, int cw) { return cw * tiles_of<QT>(nt == 1 ? 3 : 2); }  // (Q6_K: one each)

// 2 to 16 activation rows.
template <int QT, int NT>
int32_t launch_mma(tlc_ctx *ctx, GemvParams &p) {
    constexpr int TILE = QTraits<QT>::TILE_BYTES, T1 = tiles_of<QT>(1);
    const size_t budget = (size_t)ctx->prop.sharedMemPerBlockOptin;
    const size_t half = (size_t)ctx->prop.sharedMemPerMultiprocessor / 2 - 1024;
    // A warp keeps its share of the activations in registers (up to 12 blocks of K, 8 for two row
    // tiles): eight warps and two CTAs per SM hold K = 3072, sixteen warps and one CTA 6144; a
    // longer K is shared out over the CTAs of a cluster.
    const int cw = p.ktiles <= max_window<QT>(NT, 8) ? 8 : 16;
    int ks = cw == 8 ? 1 : (p.ktiles + max_window<QT>(NT, 16) - 1) / max_window<QT>(NT, 16);
    // ... over enough of them that three stages of the ring fit
    while (ks > 1 && ks < 8 && (size_t)((p.ktiles + ks - 1) / ks) * TILE > 52 * 1024) ks++;
    TLC_REQUIRE(ks <= kMaxCluster, TLC_ERR_INVALID_OPERATION, "gemv: K = %d too large", p.k);
    int max_ctas = cw == 8 ? 2 * ctx->sm_count : ctx->sm_count;
    if (ks > 1) {
        const int n = gemv_clusters(ctx, ks);
        TLC_REQUIRE(n >= 1, TLC_ERR_INVALID_OPERATION, "gemv: K = %d needs a cluster of %d CTAs", p.k, ks);
        max_ctas = n * ks;
    }
    p.ksplit = ks;
    p.ktiles_win = (p.ktiles + ks - 1) / ks;
    p.tiles_warp = (p.ktiles_win + cw - 1) / cw;
    const int ti = (p.tiles_warp + T1 - 1) / T1;
    p.stage_bytes = QT == TLC_TYPE_Q6_K ? (p.ktiles_win + 7) / 8 * kQ6Box : p.ktiles_win * TILE;
    p.m_inv = 65536 / p.m + 1;
    int grid = p.total_units * ks < max_ctas ? p.total_units * ks : max_ctas;
    const int units_per_cta = (p.total_units + grid / ks - 1) / (grid / ks);
    const size_t cap = cw == 8 ? half : budget;
    // Slabs between two cross-warp reductions, and (clusters) between two exchanges.
    int batch = NT == 1 ? 4 : 2;
    while (batch > p.subs && batch > units_per_cta * p.subs) batch /= 2;
    if (batch < p.subs) batch = p.subs;
    GemvSmem lay;
    for (;; batch /= 2) {
        p.batch = batch;
        p.round = 0;
        p.n_rounds = 1;
        if (ks > 1) {
            int round = (NT == 1 ? 64 : 32) / batch * batch;
            const int all = (units_per_cta * p.subs + batch - 1) / batch * batch;
            p.round = round < all ? round : all;
            p.n_rounds = (units_per_cta * p.subs + p.round - 1) / p.round;
        }
        lay = gemv_smem(cw, starts_of<QT>(ti), NT, p.batch, p.round);
        if ((size_t)lay.ring + 3 * (size_t)p.stage_bytes <= cap || batch <= p.subs) break;
    }
    // No more stages than this CTA will ever fill.
    const int per_cta = units_per_cta * p.subs;
    int stages = lay.ring < (int)cap ? (int)((cap - lay.ring) / p.stage_bytes) : 0;
    TLC_REQUIRE(stages >= 1, TLC_ERR_INVALID_OPERATION, "gemv: K = %d does not fit in shared memory", p.k);
    if (stages > 8) stages = 8;
    if (stages > per_cta) stages = per_cta;
    p.nstages = stages;
    // Mode 4 decides per launch.  A kernel whose CTAs stream 150 KB or more (40 MB over the grid, about 6 us
    // of HBM time) lets its successor in right after its own dependency wait: the successor is then resident
    // with its ring filled when this grid ends (Llama-70B decode: 10.07 -> 9.74 ms per token).  Shorter kernels
    // keep the late trigger (TinyLlama decode: 2.2 % slower with the early one from 54 KB on, 0.5 %
    // slower with it everywhere).
    p.pdl_mode = ctx->pdl_mode == 4 ? ((size_t)per_cta * p.stage_bytes >= 147456 ? 3 : 2) : ctx->pdl_mode;
    p.contig = units_per_cta <= 4 ? 1 : 0;
    const size_t smem = (size_t)lay.ring + (size_t)stages * p.stage_bytes;
#define TLC_GEMV_CASE(TI) \
    if (ti == TI) return cw == 8 ? launch_rows<QT, NT, TI, 8>(ctx, p, grid, smem) : launch_rows<QT, NT, TI, 16>(ctx, p, grid, smem);
    TLC_GEMV_CASE(1)
    if constexpr (QT != TLC_TYPE_Q6_K) {
        TLC_GEMV_CASE(2)
        if constexpr (NT == 1) {
            TLC_GEMV_CASE(3)
        }
    }
#undef TLC_GEMV_CASE
    return tlc_fail(TLC_ERR_INVALID_OPERATION, "gemv: K = %d too large", p.k);
}

}  // namespace

// Failure-detection self-test: a CTA waits on an mbarrier that nothing ever
// completes, through the same bounded wait the GEMV uses.  The wait runs out
// after the context's limit, the status word is set and the kernel returns.
namespace {
__global__ void selftest_mbarrier_wait_kernel(tlc_dev_status *status, uint64_t wait_ns) {
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    mbar_wait(&bar, 0, &abort_flag, status, 99, wait_ns);
}
}  // namespace

int32_t tlc_selftest_mbarrier_wait(tlc_ctx *ctx) {
    selftest_mbarrier_wait_kernel<<<1, 32, 0, ctx->stream>>>(ctx->dev_status, ctx->wait_ns);
    TLC_CHECK_LAUNCH(ctx);
    return TLC_OK;
}

int64_t tlc_gemv_max_tiles(int32_t type) {
    return kMaxCluster * (type == TLC_TYPE_Q4_0 ? max_window<TLC_TYPE_Q4_0>(1, 16) : max_window<TLC_TYPE_Q8_0>(1, 16));
}

// Scratch the RMSNorm of 2..16 rows of width k takes (their fragment order).
size_t tlc_gemv_scratch_bytes(int64_t k) { return frag_total_bytes(k / 32, 2); }

int32_t tlc_launch_gemv(tlc_ctx *ctx, const tlc_gemv_args &a) {
    TLC_REQUIRE(a.n_out >= 1 && a.n_out <= 3, TLC_ERR_INVALID_OPERATION, "gemv: %d outputs", a.n_out);
    TLC_REQUIRE(a.m >= 1, TLC_ERR_INVALID_OPERATION, "gemv: m = %d", a.m);
    const tlc_qtensor *w0 = a.outs[0].w;
    const int type = w0->type;
    const int64_t k = w0->n_cols;
    for (int i = 0; i < a.n_out; i++) {
        const tlc_qtensor *w = a.outs[i].w;
        TLC_REQUIRE(w && a.outs[i].y, TLC_ERR_INVALID_OPERATION, "gemv: null weight or output");
        TLC_REQUIRE(w->ctx->device == ctx->device, TLC_ERR_DEVICE,
                    "linear requires tensors on same device (weight on %d, context on %d)", w->ctx->device,
                    ctx->device);
        TLC_REQUIRE(w->type == type && w->n_cols == k, TLC_ERR_INVALID_OPERATION,
                    "fused linears must share type and input width");
        if (a.outs[i].rope_heads > 0)
            TLC_REQUIRE(w->n_rows % a.outs[i].rope_heads == 0 && (w->n_rows / a.outs[i].rope_heads) % 2 == 0,
                        TLC_ERR_INVALID_OPERATION, "rope needs an even head_dim (rows %lld, heads %d)",
                        (long long)w->n_rows, a.outs[i].rope_heads);
    }
    if (a.epilogue == TLC_EPI_SWIGLU)
        TLC_REQUIRE(a.n_out == 2 && a.outs[0].w->n_rows == a.outs[1].w->n_rows, TLC_ERR_INVALID_OPERATION,
                    "gate and up projections must have the same shape");

    if (type == TLC_TYPE_F16) {
        // Dense weights: RMSNorm (if asked for) runs as its own kernel, bias and
        // residual are applied in the store; RoPE, SiLU.mul and cache addressing
        // exist on the quantized path only.
        TLC_REQUIRE(a.epilogue != TLC_EPI_SWIGLU && a.n_out == 1 && a.outs[0].rope_heads == 0 &&
                        a.outs[0].row_stride < 0 && a.outs[0].pos_stride == 0,
                    TLC_ERR_INVALID_OPERATION, "fused RoPE / SiLU.mul / cache epilogues need a quantized weight");
        const __half *x = static_cast<const __half *>(a.x);
        if (a.norm_w) {
            if (int32_t rc = tlc_scratch_reserve(ctx, (size_t)a.m * k * 2)) return rc;
            if (int32_t rc = tlc_launch_rms_norm(ctx, a.x, a.norm_w, ctx->scratch, a.m, (int32_t)k, a.eps, a.norm_early)) return rc;
            x = static_cast<const __half *>(ctx->scratch);
        }
        const int threads = 256;
        const unsigned grid = (unsigned)((w0->n_rows * 32 + threads - 1) / threads);
        const __half *residual = a.epilogue == TLC_EPI_RESIDUAL ? static_cast<const __half *>(a.residual) : nullptr;
        const bool vec = k % 8 == 0 && w0->row_pitch % 16 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)w0->data % 16) == 0;
        if (a.m >= 2 && (vec || (!residual && !a.norm_w)))  // (a normalised x of odd width lies in the scratch the copies need)
            return tlc_launch_gemm_f16(ctx, w0->data, w0->row_pitch, (int)w0->n_rows, (int)k, x, a.m, a.outs[0].y,
                                       a.epilogue == TLC_EPI_STORE ? a.bias : nullptr, residual);
        if (!vec) {
            TLC_REQUIRE(!residual, TLC_ERR_INVALID_OPERATION, "residual epilogue needs 16-byte aligned f16 rows");
            linear_generic_kernel<<<grid, threads, 0, ctx->stream>>>(
                static_cast<const uint8_t *>(w0->data), w0->row_pitch, (int)w0->n_rows, (int)k, x, a.m,
                static_cast<__half *>(a.outs[0].y), static_cast<const __half *>(a.bias));
            TLC_CHECK_LAUNCH(ctx);
            return TLC_OK;
        }
        const cudaError_t le = tlc_launch_pdl(ctx, linear_f16_kernel, dim3(grid), dim3(threads), 0,
                                              static_cast<const uint8_t *>(w0->data), w0->row_pitch, (int)w0->n_rows, (int)k, x,
                                              static_cast<__half *>(a.outs[0].y), static_cast<const __half *>(a.bias), residual);
        if (le != cudaSuccess) {
            cudaGetLastError();
            return tlc_fail(TLC_ERR_CUDA, "f16 linear launch failed: %s", cudaGetErrorString(le));
        }
        TLC_CHECK_LAUNCH(ctx);
        return TLC_OK;
    }

    if (type == TLC_TYPE_Q6_K) {
        // Resident Q6_K (stock Q4_0 GGUF files store output.weight, the largest linear of a decode step, so): one
        // weight per launch; RMSNorm, if asked for, as its own kernel; bias and residual in the store.
        // More than sixteen activation rows take further passes.  Bound by the integer operations that put the 4 + 2
        // bits together (ten an MMA of 16 x 16 weights), at about half of the HBM rate.
        TLC_REQUIRE(a.epilogue != TLC_EPI_SWIGLU && a.n_out == 1 && a.outs[0].rope_heads == 0 &&
                        a.outs[0].row_stride < 0 && a.outs[0].pos_stride == 0,
                    TLC_ERR_INVALID_OPERATION, "fused RoPE / SiLU.mul / cache epilogues need a Q4_0 or Q8_0 weight");
        const __half *x = static_cast<const __half *>(a.x);
        if (a.norm_w) {
            if (int32_t rc = tlc_scratch_reserve(ctx, (size_t)a.m * k * 2)) return rc;
            if (int32_t rc = tlc_launch_rms_norm(ctx, a.x, a.norm_w, ctx->scratch, a.m, (int32_t)k, a.eps, a.norm_early)) return rc;
            x = static_cast<const __half *>(ctx->scratch);
        }
        TLC_REQUIRE(((uintptr_t)x & 15) == 0, TLC_ERR_INVALID_OPERATION, "linear: activations must be 16-byte aligned");
        if (k / 256 > kMaxCluster * max_window<TLC_TYPE_Q6_K>(1, 16)) {
            const cudaError_t le = tlc_launch_pdl(ctx, linear_q6k_long_kernel, dim3((unsigned)((w0->n_rows + 7) / 8)), dim3(256), 0,
                                                  static_cast<const uint8_t *>(w0->data), w0->row_pitch, (int)w0->n_rows, (int)k, x, a.m,
                                                  static_cast<__half *>(a.outs[0].y), static_cast<const __half *>(a.bias),
                                                  a.epilogue == TLC_EPI_RESIDUAL ? static_cast<const __half *>(a.residual) : nullptr);
            if (le != cudaSuccess) {
                cudaGetLastError();
                return tlc_fail(TLC_ERR_CUDA, "Q6_K linear launch failed: %s", cudaGetErrorString(le));
            }
            TLC_CHECK_LAUNCH(ctx);
            return TLC_OK;
        }
        // (Sixteen rows cost 1.6 times eight, so passes of sixteen: 32000 x 2048 at 17 / 19 / 24 / 32 rows takes 43.2 / 43.5 /
        // 45.3 / 54.5 us, in passes of eight 50.4 / 50.9 / 52.3 / 69.3.)
        constexpr int pass = 16;
        for (int m0 = 0; m0 < a.m; m0 += pass) {
            GemvParams p{};
            p.m = a.m - m0 < pass ? a.m - m0 : pass;
            p.n_out = 1;
            p.subs = 1;
            p.t[0].n = (int)w0->n_rows;
            p.t[0].row_stride = w0->n_rows;
            p.t[0].y = static_cast<__half *>(a.outs[0].y) + (size_t)m0 * w0->n_rows;
            p.slabs[0] = p.total_units = (int)((w0->n_rows + kRows - 1) / kRows);
            p.k = (int)k;
            p.nblk = (int)(k / 16);
            p.ktiles = (int)(k / 256);
            p.x = x + (size_t)m0 * k;
            p.epilogue = a.epilogue;
            p.bias = static_cast<const __half *>(a.bias);
            p.residual = a.epilogue == TLC_EPI_RESIDUAL ? static_cast<const __half *>(a.residual) + (size_t)m0 * w0->n_rows : nullptr;
            p.status = ctx->dev_status;
            p.wait_ns = ctx->wait_ns;
            CUtensorMap map;
            static_assert(sizeof map == sizeof p.w_map, "tensor map size");
            TLC_REQUIRE(tlc_gemm::encode_map(&map, CU_TENSOR_MAP_DATA_TYPE_UINT64, CU_TENSOR_MAP_SWIZZLE_NONE, w0->data, w0->row_pitch / 8,
                                             (uint64_t)w0->n_rows, w0->row_pitch, kQ6BoxRow / 8, kRows),
                        TLC_ERR_CUDA, "linear: no tensor map for a Q6_K weight");
            memcpy(p.w_map, &map, sizeof map);
            if (int32_t rc = p.m <= 8 ? launch_mma<TLC_TYPE_Q6_K, 1>(ctx, p) : launch_mma<TLC_TYPE_Q6_K, 2>(ctx, p)) return rc;
        }
        return TLC_OK;
    }

    if (tlc_gemm_eligible(ctx, a)) return tlc_launch_gemm(ctx, a);

    // (a lane's eight values of a block: two 8-byte pieces of Q4_0, one of 16 bytes of Q8_0)
    TLC_REQUIRE((((uintptr_t)a.x | (uintptr_t)a.norm_w) & (type == TLC_TYPE_Q4_0 ? 7 : 15)) == 0, TLC_ERR_INVALID_OPERATION,
                "linear: activations and norm weights must be %d-byte aligned", type == TLC_TYPE_Q4_0 ? 8 : 16);
    // (more than sixteen rows, where tlc_gemm_eligible leaves them here: passes over the weights)
    const int64_t nt2_tiles = kMaxCluster * (type == TLC_TYPE_Q4_0 ? max_window<TLC_TYPE_Q4_0>(2, 16) : max_window<TLC_TYPE_Q8_0>(2, 16));
    // (the longest K: even passes of up to eight rows, not eight and a last one, which the one-row kernel cannot hold)
    const int passes = (a.m + 7) / 8, max_m = w0->k_tiles <= nt2_tiles ? 16 : (a.m + passes - 1) / passes;
    for (int m0 = 0; m0 < a.m; m0 += max_m) {
        const int mc = a.m - m0 < max_m ? a.m - m0 : max_m;
        GemvParams p{};
        p.n_out = a.n_out;
        p.total_units = 0;
        for (int i = 0; i < a.n_out; i++) {
            const tlc_qtensor *w = a.outs[i].w;
            p.t[i].w = static_cast<const uint8_t *>(w->data);
            p.t[i].slab_pitch = w->slab_pitch;
            p.t[i].n = (int)w->n_rows;
            // Outputs are [m, N] row-major: a pass over rows m0.. writes at y + m0*N.
            const long long rs = a.outs[i].row_stride >= 0 ? a.outs[i].row_stride : (long long)w->n_rows;
            p.t[i].row_stride = rs;
            p.t[i].pos_stride = a.outs[i].pos_stride;
            p.t[i].y = static_cast<__half *>(a.outs[i].y) + (size_t)m0 * rs;
            p.t[i].rope_heads = a.outs[i].rope_heads;
            p.t[i].head_dim = a.outs[i].rope_heads > 0 ? (int)(w->n_rows / a.outs[i].rope_heads) : 0;
            p.slabs[i] = (int)((w->n_rows + kRows - 1) / kRows);
            p.total_units += p.slabs[i];
        }
        p.subs = 1;
        if (a.epilogue == TLC_EPI_SWIGLU) {
            p.subs = 2;
            p.total_units = p.slabs[0];
        }
        p.k = (int)k;
        p.nblk = (int)(k / 32);
        p.ktiles = (int)w0->k_tiles;
        p.m = mc;
        p.x = static_cast<const __half *>(a.x) + (size_t)m0 * k;
        p.norm_w = static_cast<const __half *>(a.norm_w);
        p.norm_early = a.norm_early ? 1 : 0;
        p.eps = a.eps;
        p.epilogue = a.epilogue;
        p.bias = static_cast<const __half *>(a.bias);
        p.residual = a.residual ? static_cast<const __half *>(a.residual) + (size_t)m0 * w0->n_rows : nullptr;
        p.pos_offset = a.pos_offset + m0;
        p.rope_base = (float)a.rope_base;
        p.positions = a.positions ? a.positions + m0 : nullptr;
        p.max_pos = a.max_pos;
        p.status = ctx->dev_status;
        p.wait_ns = ctx->wait_ns;
        const int nt = mc > 8 ? 2 : 1;
        const bool q4 = type == TLC_TYPE_Q4_0;
        if (mc > 1 && a.norm_w) {
            const int64_t nblk = k / 32;
            if (int32_t rc = tlc_scratch_reserve(ctx, frag_total_bytes(nblk, nt))) return rc;
            uint4 *frag = static_cast<uint4 *>(ctx->scratch);
            float *start = reinterpret_cast<float *>(static_cast<uint8_t *>(ctx->scratch) + frag_bytes(nblk, nt));
            auto *fn = a.norm_early ? (q4 ? frag_rows_kernel<TLC_TYPE_Q4_0, true> : frag_rows_kernel<TLC_TYPE_Q8_0, true>)
                                    : (q4 ? frag_rows_kernel<TLC_TYPE_Q4_0, false> : frag_rows_kernel<TLC_TYPE_Q8_0, false>);
            const cudaError_t le = tlc_launch_pdl(ctx, fn, dim3(8 * nt), dim3(512), 0, p.x, p.norm_w, mc, (int)k, a.eps, frag, start, nt);
            if (le != cudaSuccess) {
                cudaGetLastError();
                return tlc_fail(TLC_ERR_CUDA, "gemv: RMSNorm launch failed: %s", cudaGetErrorString(le));
            }
            TLC_CHECK_LAUNCH(ctx);
            p.frag = frag;
            p.start = start;
            p.norm_w = nullptr;
        }
        int32_t rc;
        if (mc == 1)
            rc = q4 ? launch_row1<TLC_TYPE_Q4_0>(ctx, p) : launch_row1<TLC_TYPE_Q8_0>(ctx, p);
        else if (q4)
            rc = nt == 1 ? launch_mma<TLC_TYPE_Q4_0, 1>(ctx, p) : launch_mma<TLC_TYPE_Q4_0, 2>(ctx, p);
        else
            rc = nt == 1 ? launch_mma<TLC_TYPE_Q8_0, 1>(ctx, p) : launch_mma<TLC_TYPE_Q8_0, 2>(ctx, p);
        if (rc) return rc;
    }
    return TLC_OK;
}
