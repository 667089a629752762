// Kernel body and launcher of the tcgen05 dequant-GEMM (see tlc_gemm_kernel.cuh).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <climits>
#include <type_traits>

#include "tlc_gemm_kernel.cuh"
#include "tlc_gemm_wt.h"

using namespace tlc_gemm;

// Tensor map of a row-major matrix [outer, inner], rows `pitch` bytes apart: boxes of box_outer rows x
// box_inner elements, zero fill outside.  False when the driver entry point is missing or refuses the shape.
// Extents and box from the contiguous dimension outwards; `pitches`: bytes from one element to the next of
// each dimension but that one.
bool tlc_gemm::encode_map_nd(CUtensorMap *map, CUtensorMapDataType type, CUtensorMapSwizzle swizzle, const void *ptr,
                             int rank, const uint64_t *dims, const uint64_t *pitches, const uint32_t *box) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess)
            fn = nullptr;
        cudaGetLastError();
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }();
    if (!encode || ((uintptr_t)ptr & 15) != 0) return false;
    cuuint64_t d[5], st[4];
    cuuint32_t bx[5], es[5];
    for (int i = 0; i < rank; i++) {
        d[i] = dims[i];
        bx[i] = box[i];
        es[i] = 1;
        if (i + 1 < rank) {
            if ((pitches[i] & 15) != 0) return false;
            st[i] = pitches[i];
        }
    }
    return encode(map, type, (cuuint32_t)rank, const_cast<void *>(ptr), d, st, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool tlc_gemm::encode_map(CUtensorMap *map, CUtensorMapDataType type, CUtensorMapSwizzle swizzle, const void *ptr,
                          uint64_t inner, uint64_t outer, uint64_t pitch, uint32_t box_inner, uint32_t box_outer) {
    const uint64_t dims[2] = {inner, outer};
    const uint32_t box[2] = {box_inner, box_outer};
    return encode_map_nd(map, type, swizzle, ptr, 2, dims, &pitch, box);
}

bool tlc_gemm::encode_f16_map(CUtensorMap *map, const void *ptr, uint64_t inner, uint64_t outer, uint64_t pitch,
                              uint32_t box_inner, uint32_t box_outer) {
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, ptr, inner, outer, pitch, box_inner,
                      box_outer);
}

// Tensor map of the activations [M, K] for the 128-row tiles of this file; the cp.async loaders take
// over when there is none.
bool tlc_gemm::encode_x_map(CUtensorMap *map, const GemmParams &p) {
    return encode_f16_map(map, p.x, (uint64_t)p.k, (uint64_t)p.m, (uint64_t)p.k * 2, kBK, 128);
}

namespace {

// B producer of one weight row.  The row's share of a weight tile (64 bytes of
// quants: four 16-byte pieces, plus its block scales) covers two K steps for
// Q4_0 and one for Q8_0; shares are fetched in groups of two tiles, one group
// ahead of their use, so the global-memory latency is spread over a group's
// worth of K steps.
template <int QT, int STAGES, int STAGE_BYTES>
__device__ __forceinline__ void produce_b(const GemmParams &p, uint8_t *btiles, uint64_t *full, uint64_t *empty,
                                          volatile int *abort_flag, const uint8_t *wbase, int wrow, int row, int KT,
                                          int lane) {
    constexpr int TILE = QT == TLC_TYPE_Q4_0 ? 1152 : 1088;
    constexpr int TS = QT == TLC_TYPE_Q4_0 ? 2 : 1;  // K steps per tile
    constexpr int GT = 2;                             // tiles per group
    // `row`: row of the smem tile this thread fills; `wrow`: the weight row it holds (of `wbase`).
    // Rows past N load nothing: a zero scale makes every value of the tile row zero.
    const bool row_ok = wrow < p.n;
    const int r16 = wrow & 15;
    const uint8_t *slab = wbase + (size_t)(row_ok ? wrow >> 4 : 0) * p.w_pitch;
    const uint32_t qoff = (uint32_t)((r16 >> 3) * 512 + (r16 & 7) * 64);
    const uint32_t soff = 1024u + (uint32_t)r16 * (QT == TLC_TYPE_Q4_0 ? 8u : 4u);
    uint4 nxt4[GT * 4], cur4[GT * 4];
    uint32_t nxts[GT * TS], curs[GT * TS];
    auto load_group = [&](int g) {
#pragma unroll
        for (int i = 0; i < GT; i++) {
            const int kt = g * GT + i;
            const bool ok = row_ok && kt < p.k_tiles;
            const uint8_t *tile = slab + (size_t)(ok ? kt : 0) * TILE;
#pragma unroll
            for (int t = 0; t < 4; t++)
                nxt4[i * 4 + t] = ok ? __ldg(reinterpret_cast<const uint4 *>(tile + qoff) + t) : make_uint4(0, 0, 0, 0);
            if (QT == TLC_TYPE_Q4_0) {
                const uint2 sc = ok ? __ldg(reinterpret_cast<const uint2 *>(tile + soff)) : make_uint2(0, 0);
                nxts[i * TS] = sc.x;
                nxts[i * TS + TS - 1] = sc.y;
            } else {
                nxts[i * TS] = ok ? __ldg(reinterpret_cast<const uint32_t *>(tile + soff)) : 0u;
            }
        }
    };
    // byte offsets of the eight 16-byte pieces of this row under the 128-byte swizzle
    uint32_t piece[8];
#pragma unroll
    for (int j = 0; j < 8; j++) piece[j] = (uint32_t)(row * 128 + ((j ^ (row & 7)) << 4));
    constexpr int SPG = GT * TS;  // K steps per group
    const int n_groups = (KT + SPG - 1) / SPG;
    auto comp = [](const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; };
    auto process = [&](int g) {
#pragma unroll
        for (int st = 0; st < SPG; st++) {
            const int kt = g * SPG + st;
            if (kt >= KT) break;
            const int ti = st / TS;        // tile of the group
            const int half = st % TS;      // Q4_0: which pair of the tile's four blocks
            const uint32_t scw = curs[ti * TS + half];  // the two scales of this K step
            const int s = kt % STAGES;
            mbar_wait(&empty[s], ((kt / STAGES) & 1u) ^ 1u, abort_flag, p.status, 11, p.wait_ns);
            uint8_t *bt = btiles + (size_t)s * STAGE_BYTES;
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const __half d = __ushort_as_half((unsigned short)(e == 0 ? scw & 0xFFFFu : scw >> 16));
                if (QT == TLC_TYPE_Q4_0) {
                    uint32_t q[4];
#pragma unroll
                    for (int t = 0; t < 4; t++) q[t] = comp(cur4[ti * 4 + t], 2 * half + e);
                    dequant_block<QT>(q, d, bt, piece, e);
                } else {
                    uint32_t q[8];
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        q[2 * t] = comp(cur4[ti * 4 + t], 2 * e);
                        q[2 * t + 1] = comp(cur4[ti * 4 + t], 2 * e + 1);
                    }
                    dequant_block<QT>(q, d, bt, piece, e);
                }
            }
            fence_async_proxy();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    };
    load_group(0);
#pragma unroll 1
    for (int g = 0; g < n_groups; g++) {
#pragma unroll
        for (int i = 0; i < GT * 4; i++) cur4[i] = nxt4[i];
#pragma unroll
        for (int i = 0; i < GT * TS; i++) curs[i] = nxts[i];
        if (g + 1 < n_groups) load_group(g + 1);
        process(g);
    }
}

// SW: the SiLU.mul pair.  The weight tile holds 128 rows of the gate weight (tile rows
// 0-127) and the same 128 rows of the up weight (tile rows 128-255); the epilogue reads
// both accumulators and stores silu(gate) * up for the 128 output columns of the CTA.
template <int QT, int MT, int NT, bool SW>
__global__ void __launch_bounds__(gemm_threads(NT), 1)
    gemm_tcgen05_kernel(const GemmParams p, const __grid_constant__ CUtensorMap x_map) {
    static_assert(!SW || NT == 2, "the gate/up pair fills a 256-row weight tile");
    constexpr int BN = 128 * NT;
    constexpr int A_BYTES = 128 * MT * 128, B_BYTES = BN * 128;
    constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr int kStages = stages_for(MT, NT);
    constexpr uint32_t TMEM_COLS = MT * BN;  // 128, 256 or 512: a power of two
    constexpr uint32_t IDESC = idesc_for(BN);
    constexpr int MMA_WARP = 4 + 4 * NT;

    extern __shared__ uint8_t smem_raw[];
    uint8_t *tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *full = reinterpret_cast<uint64_t *>(tiles + (size_t)kStages * STAGE_BYTES);
    uint64_t *empty = full + kStages;
    uint64_t *accum_bar = empty + kStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accum_bar + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int n0 = blockIdx.x * (SW ? 128 : BN), m0 = blockIdx.y * 128 * MT;
    const int KT = (p.k + kBK - 1) / kBK;  // K is a multiple of 32: the last step may hold one block only

    if (tid == 0) {
        for (int s = 0; s < kStages; s++) {
            // the activation tile arrives by TMA (one arrive.expect_tx) or from the four
            // cp.async loader warps; the working B-producer warps arrive once each
            mbar_init(&full[s], (p.a_tma ? 1 : 4) + 4 * NT);
            mbar_init(&empty[s], 1);          // tcgen05.commit
        }
        mbar_init(accum_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    tlc_pdl_prologue();  // x (and residual) come from the previous kernel of the stream

    if (warp >= 4 && warp < MMA_WARP) {
        const int trow = (tid - 128) % BN;  // row of the weight tile
        const uint8_t *wbase = SW && trow >= 128 ? p.w2 : p.w;
        const int wrow = SW ? n0 + (trow & 127) : n0 + trow;
        produce_b<QT, kStages, STAGE_BYTES>(p, tiles + A_BYTES, full, empty, abort_flag, wbase, wrow, trow, KT, lane);
    } else if (warp < 4 && p.a_tma) {
        // ------------------------------ A tile by TMA ------------------------------
        // One warp issues, per K step, MT boxes of 128 rows x 64 columns with the 128-byte
        // swizzle of the tile; rows past M and columns past K read the zero fill.  The
        // inner coordinate is a multiple of 64 elements (128 bytes).
        if (warp == 0) {
            const uint32_t el = elect_one();
            if (el) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&x_map)) : "memory");
            int s = 0;
            uint32_t ph = 1;
            for (int j = 0; j < KT; j++) {
                if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ph, abort_flag, p.status, 12, p.wait_ns))) break;
                const uint32_t bar = smem_u32(&full[s]);
                const uint32_t abase = smem_u32(tiles + (size_t)s * STAGE_BYTES);
                mbar_arrive_expect_tx_el(&full[s], A_BYTES, el);
#pragma unroll
                for (int i = 0; i < MT; i++)
                    tma_load_2d_el(abase + i * (128 * 128), &x_map, j * kBK, m0 + 128 * i, bar, el);
                if (++s == kStages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp < 4) {
        // ------------------------------ A loaders (cp.async) ------------------------------
        auto issue = [&](int j) {
            const int s = j % kStages;
            mbar_wait(&empty[s], ((j / kStages) & 1u) ^ 1u, abort_flag, p.status, 12, p.wait_ns);
            const uint32_t abase = smem_u32(tiles + (size_t)s * STAGE_BYTES);
            // 8 consecutive threads copy the 128 bytes of one row.
#pragma unroll
            for (int it = 0; it < 8 * MT; it++) {
                const int row = it * 16 + (tid >> 3), c = tid & 7;
                // rows past M and, in a last step of one block, columns past K are zero-filled
                const bool ok = m0 + row < p.m && j * kBK + c * 8 < p.k;
                const __half *src = p.x + (ok ? (size_t)(m0 + row) * p.k + (size_t)j * kBK + c * 8 : 0);
                cp_async16(abase + row * 128 + ((c ^ (row & 7)) << 4), src, ok);
            }
        };
        constexpr int kAhead = kStages - 1;
        for (int j = 0; j < kAhead; j++) {
            if (j < KT) issue(j);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        for (int kt = 0; kt < KT; kt++) {
            // Hand over stage kt first, then refill the stage the MMA of step
            // kt-1 is about to free: the hand-over must not wait for that MMA.
            asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
            fence_async_proxy();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[kt % kStages]);
            const int j = kt + kAhead;
            if (j < KT) issue(j);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    } else if (warp == MMA_WARP) {
        // ------------------------------ MMA issuer ------------------------------
        const uint32_t el = elect_one();
        const uint32_t a0 = (smem_u32(tiles) & 0x3FFFF) >> 4;
        int s = 0;
        uint32_t ph = 0, acc = 0;
        for (int kt = 0; kt < KT; kt++) {
            const bool ready = __all_sync(0xffffffffu, mbar_wait(&full[s], ph, abort_flag, p.status, 14, p.wait_ns));
            tc_fence_after();
            if (ready) {
                const uint32_t a_addr = a0 + (uint32_t)s * (STAGE_BYTES >> 4), b_addr = a_addr + (A_BYTES >> 4);
#pragma unroll
                for (int k16 = 0; k16 < kBK / 16; k16++) {
#pragma unroll
                    for (int i = 0; i < MT; i++)
                        umma_f16(tmem_base + BN * i, desc_at(a_addr + i * ((128 * 128) >> 4) + k16 * 2),
                                 desc_at(b_addr + k16 * 2), IDESC, acc, el);
                    acc = 1;
                }
            }
            umma_commit(&empty[s], el);  // arrives when the MMAs above have read the stage
            if (++s == kStages) {
                s = 0;
                ph ^= 1u;
            }
        }
        umma_commit(accum_bar, el);
        __syncwarp();
    }

    // ------------------------------ epilogue ------------------------------
    // Warp w reads tensor-memory lanes 32*(w%4) .. +31 (= activation rows of a
    // sub-tile); the warps of a lane quarter (two or three) take the 32-column pieces in turn.
    if (warp < MMA_WARP) {
        mbar_wait(accum_bar, 0, abort_flag, p.status, 13, p.wait_ns);
        __syncwarp();  // the lanes leave a wait one by one; tcgen05.ld is for a whole warp
        tc_fence_after();
        const int wq = warp & 3;
        constexpr int OUT_COLS = SW ? 128 : BN;  // output columns of the CTA
        constexpr int PIECES = MT * OUT_COLS / 32;
#pragma unroll 1
        for (int pc = warp >> 2; pc < PIECES; pc += MMA_WARP / 4) {
            __syncwarp();
            const int i = pc / (OUT_COLS / 32), c0 = (pc % (OUT_COLS / 32)) * 32;
            const int row = m0 + 128 * i + 32 * wq + lane;
            bool row_ok = row < p.m;
            const int pos = !row_ok ? 0 : p.positions ? p.positions[row] : p.pos_offset + row;
            if (row_ok && p.pos_stride != 0 && p.max_pos > 0 && (pos < 0 || pos >= p.max_pos)) {
                // a cache row that does not exist: nothing is written, the host hears about it
                if (atomicCAS(&p.status->code, 0, TLC_DEV_INDEX) == 0) p.status->where = 301;
                row_ok = false;
            }
            // Dense rows by default; a KV-cache destination addresses rows by (sequence, position).
            __half *ybase = p.y + (size_t)((long long)row * p.row_stride + (long long)pos * p.pos_stride);
            uint32_t r[32];
            tmem_ld32(tmem_base + ((uint32_t)(32 * wq) << 16) + (uint32_t)(BN * i + c0), r);
            if (SW) {
                // s = sigmoid(g) (f32, RNE); a = g*s; act = a*u: three f16 roundings as in
                // debug/chat_demo_with_kvcache.tl:26-41 (the GEMV's SiLU.mul epilogue does the same)
                uint32_t ru[32];
                tmem_ld32(tmem_base + ((uint32_t)(32 * wq) << 16) + (uint32_t)(BN * i + 128 + c0), ru);
                if (row_ok && n0 + c0 < p.n) epilogue_piece_swiglu(p, r, ru, n0 + c0, ybase);
            } else if (row_ok && n0 + c0 < p.n) {
                epilogue_piece(p, r, row, pos, n0 + c0, ybase);
            }
        }
        tc_fence_before();
    }

    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

template <int QT, int MT, int NT, bool SW = false>
int32_t launch_tile(tlc_ctx *ctx, const GemmParams &p) {
    const size_t smem = smem_bytes(MT, NT);
    static bool configured[64] = {};
    if (!configured[ctx->device & 63]) {
        TLC_CUDA(cudaFuncSetAttribute(gemm_tcgen05_kernel<QT, MT, NT, SW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        TLC_CUDA(cudaFuncSetAttribute(gemm_tcgen05_kernel<QT, MT, NT, SW>,
                                      cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        configured[ctx->device & 63] = true;
    }
    const int out_cols = SW ? 128 : 128 * NT;  // output columns per CTA
    GemmParams q = p;
    const dim3 grid((unsigned)((p.n + out_cols - 1) / out_cols), (unsigned)((p.m + 128 * MT - 1) / (128 * MT)));
    CUtensorMap x_map;
    memset(&x_map, 0, sizeof x_map);
    q.a_tma = ctx->gemm_tma && encode_x_map(&x_map, p) ? 1 : 0;
    cudaError_t le = tlc_launch_pdl(ctx, gemm_tcgen05_kernel<QT, MT, NT, SW>, grid, dim3(gemm_threads(NT)), smem, q,
                                    x_map);
    if (le != cudaSuccess) {
        cudaGetLastError();
        return tlc_fail(TLC_ERR_CUDA, "gemm launch failed: %s", cudaGetErrorString(le));
    }
    TLC_CHECK_LAUNCH(ctx);
    return TLC_OK;
}

template <int QT>
int32_t launch_one_t(tlc_ctx *ctx, const GemmParams &p) {
    // Tile choice: 256 x 256 halves the activation traffic from L2 per MMA against 128 x 128
    // (measured on wide weights: about 930 / 760 / 580 TFLOP/s for 256x256 / 128x256 / 128x128),
    // but a tile shape only pays if its CTAs fill the SMs: score = relative tile speed x the
    // fraction of SM slots the last wave leaves busy.
    auto ctas = [&](int mt, int nt) {
        return (long)((p.n + 128 * nt - 1) / (128 * nt)) * ((p.m + 128 * mt - 1) / (128 * mt));
    };
    auto score = [&](int mt, int nt, double speed) {
        const long c = ctas(mt, nt), sms = ctx->sm_count;
        return speed * (double)c / (double)(((c + sms - 1) / sms) * sms);
    };
    int tile = ctx->gemm_tile;  // 0: choose; 11 / 12 / 22: forced (tests)
    if (tile == 0) {
        const double s22 = p.m > 128 ? score(2, 2, 1.0) : 0.0, s12 = score(1, 2, 0.8), s11 = score(1, 1, 0.6);
        tile = s22 >= s12 && s22 >= s11 ? 22 : s12 >= s11 ? 12 : 11;
    }
    if (tile == 22) return launch_tile<QT, 2, 2>(ctx, p);
    if (tile == 12) return launch_tile<QT, 1, 2>(ctx, p);
    return launch_tile<QT, 1, 1>(ctx, p);
}

// The gate/up pair: 128 output columns per CTA (a 256-row weight tile), one or two token sub-tiles.
template <int QT>
int32_t launch_pair_t(tlc_ctx *ctx, const GemmParams &p) {
    auto ctas = [&](int mt) { return (long)((p.n + 127) / 128) * ((p.m + 128 * mt - 1) / (128 * mt)); };
    auto score = [&](int mt, double speed) {
        const long c = ctas(mt), sms = ctx->sm_count;
        return speed * (double)c / (double)(((c + sms - 1) / sms) * sms);
    };
    const bool two = ctx->gemm_tile == 22 || (ctx->gemm_tile == 0 && p.m > 128 && score(2, 1.0) >= score(1, 0.8));
    return two ? launch_tile<QT, 2, 2, true>(ctx, p) : launch_tile<QT, 1, 2, true>(ctx, p);
}

int32_t launch_one(tlc_ctx *ctx, const GemmParams &p, int type) {
    // From 129 activation rows on, two SMs share a 256 x 256 tile (tlc_gemm_pair.cu).
    if (cta_pair_eligible(ctx, p)) return launch_cta_pair(ctx, p, type, p.w2 != nullptr);
    if (p.w2) return type == TLC_TYPE_Q4_0 ? launch_pair_t<TLC_TYPE_Q4_0>(ctx, p) : launch_pair_t<TLC_TYPE_Q8_0>(ctx, p);
    return type == TLC_TYPE_Q4_0 ? launch_one_t<TLC_TYPE_Q4_0>(ctx, p) : launch_one_t<TLC_TYPE_Q8_0>(ctx, p);
}

inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace

// Context scratch the GEMM form of a linear over m rows of width k may need: the normalised rows.
// Callers that capture graphs reserve it up front.
size_t tlc_gemm_scratch_bytes(int m, int64_t k) { return align256((size_t)m * k * 2); }

bool tlc_gemm_eligible(const tlc_ctx *ctx, const tlc_gemv_args &a) {
    const tlc_qtensor *w0 = a.outs[0].w;
    if (w0->type != TLC_TYPE_Q4_0 && w0->type != TLC_TYPE_Q8_0) return false;
    // K in whole blocks; an odd block count ends in a K step whose second block is the row's
    // zero padding (rows are padded to 16 bytes with zeros at upload) against zero-filled activations
    if (w0->n_cols % 32 != 0 || w0->n_cols < kBK) return false;
    if (ctx->gemm_min_m > 0) return a.m >= ctx->gemm_min_m;
    // Up to 16 rows one pass of the GEMV reads the weights once and multiplies d * (q - 8) as it is; the GEMM
    // multiplies that rounded to f16.  With a long K the GEMM would be faster from 9 rows on (Q4_0 4096 x 11008 at 9 / 16
    // rows 15.2 us, GEMV 18.1 / 19.8; 1280 x 8192 at 16 rows 8.0 and 11.5), but against 64 bits its results are off
    // by 2.8e-4 (Q8_0 2.9e-4) where the GEMV's are by 2.1e-4, the rounding of the output: precision goes first.
    // For the same reason 17 to 48 rows stay in passes of sixteen where they have always been so, and their callers have
    // exact weights: outputs of less than half a wave of 128-row tiles, and a K that is short, or short for the
    // number of products, or so many outputs together that a wave has no room to share K out.  (8192 x 1024 at 17 /
    // 32 / 48 rows 10.4 / 12.6 / 19.4 us, GEMM 7.3 / 7.4 / 7.7; 2048 x 512 at 17 rows 6.6, GEMM 6.2.)
    // Nine and more rows of a K that no cluster of the GEMV holds the activations of (98304) have nowhere else to go.
    if (a.m > 48 || (a.m > 8 && w0->k_tiles > tlc_gemv_max_tiles(w0->type))) return true;
    if (a.m <= 16) return false;
    const bool pair = a.epilogue == TLC_EPI_SWIGLU;
    int64_t widest = 0, outputs = 0, tiles = 0;
    for (int i = 0; i < a.n_out; i++) {
        const int64_t n = a.outs[i].w->n_rows;
        widest = n > widest ? n : widest;
        outputs += n;
        tiles += pair ? (n + 127) / 128 * (i == 0) : (n + 255) / 256;
    }
    const bool exact = (widest + 127) / 128 * 2 < ctx->sm_count &&
                       (tiles * 2 > ctx->sm_count || a.m * outputs >= 650 * (w0->n_cols - 1216));
    return !exact;
}

// Same contract as tlc_launch_gemv for m activation rows on the tensor cores:
// the RMSNorm prologue runs as its own kernel into scratch, every output of a
// fused multi-projection is its own GEMM, and the SiLU.mul pair is one GEMM whose
// weight tile holds gate and up rows side by side.
int32_t tlc_launch_gemm(tlc_ctx *ctx, const tlc_gemv_args &a) {
    const tlc_qtensor *w0 = a.outs[0].w;
    const int64_t k = w0->n_cols;
    const bool swiglu = a.epilogue == TLC_EPI_SWIGLU;
    // Which form: the one with 128 activation rows on the M side of the MMA (this file) moves half the
    // activation bytes per MMA, but only in 256 x 256 tiles, and pays off where these fill the waves of SMs:
    // 8192 -> 28672 at 256 rows (112 tiles) 112 us against 134, 4096 -> 4096 at 2048 rows (128) 57 against
    // 64; but 4096 -> 11008 at 1024 rows (172 tiles, 58 % of two waves) 124 us against 100.
    // (An option that forces a detail of that form asks for the form.)
    bool wt = a.m <= ctx->gemm_wt_max_m && ctx->gemm_tile == 0 && !ctx->gemm_pair && ctx->gemm_tma;
    if (wt && ctx->gemm_wt_max_m == INT_MAX && a.m >= 192) {
        int64_t tiles = 0;
        for (int i = 0; i < a.n_out; i++) tiles = tiles > a.outs[i].w->n_rows ? tiles : a.outs[i].w->n_rows;
        tiles = ((tiles + (swiglu ? 127 : 255)) / (swiglu ? 128 : 256)) * ((a.m + 255) / 256);
        const int64_t slots = (tiles + ctx->sm_count - 1) / ctx->sm_count * ctx->sm_count;
        wt = tiles < 100 || tiles * 10 < slots * 7;
    }
    const __half *x = static_cast<const __half *>(a.x);
    if (a.norm_w) {
        if (int32_t rc = tlc_scratch_reserve(ctx, tlc_gemm_scratch_bytes(a.m, k))) return rc;
        if (int32_t rc = tlc_launch_rms_norm(ctx, a.x, a.norm_w, ctx->scratch, a.m, (int32_t)k, a.eps, a.norm_early)) return rc;
        x = static_cast<const __half *>(ctx->scratch);
    }
    TLC_REQUIRE(((uintptr_t)x & 15) == 0, TLC_ERR_INVALID_OPERATION, "gemm: activations must be 16-byte aligned");
    if (wt) {
        tlc_gemv_args b = a;
        b.x = x;
        b.norm_w = nullptr;
        return tlc_launch_gemm_wt(ctx, b);
    }
    // The SiLU.mul pair is ONE launch: gate and up rows share the weight tile of a CTA.
    const int n_launch = swiglu ? 1 : a.n_out;
    for (int i = 0; i < n_launch; i++) {
        const tlc_qtensor *w = a.outs[i].w;
        GemmParams p{};
        p.w = static_cast<const uint8_t *>(w->data);
        p.w_pitch = w->slab_pitch;
        p.k_tiles = (int)w->k_tiles;
        p.x = x;
        p.m = a.m;
        p.n = (int)w->n_rows;
        p.k = (int)k;
        p.status = ctx->dev_status;
        p.wait_ns = ctx->wait_ns;
        p.y = static_cast<__half *>(a.outs[i].y);
        if (swiglu) {
            TLC_REQUIRE(a.outs[1].w->slab_pitch == w->slab_pitch, TLC_ERR_SHAPE_MISMATCH,
                        "gate and up projections must have the same layout");
            p.w2 = static_cast<const uint8_t *>(a.outs[1].w->data);
            p.row_stride = p.n;
        } else {
            p.row_stride = a.outs[i].row_stride >= 0 ? a.outs[i].row_stride : (long long)w->n_rows;
            p.pos_stride = a.outs[i].pos_stride;
            p.head_dim = a.outs[i].rope_heads > 0 ? (int)(w->n_rows / a.outs[i].rope_heads) : 0;
            p.residual = a.epilogue == TLC_EPI_RESIDUAL ? static_cast<const __half *>(a.residual) : nullptr;
            p.bias = a.epilogue == TLC_EPI_STORE ? static_cast<const __half *>(a.bias) : nullptr;
        }
        p.pos_offset = a.pos_offset;
        p.positions = a.positions;
        p.max_pos = a.max_pos;
        p.rope_base = (float)a.rope_base;
        p.vec_ok = ((p.row_stride | p.pos_stride | (long long)p.n) & 7) == 0 && ((uintptr_t)p.y & 15) == 0 &&
                   ((uintptr_t)p.residual & 15) == 0;
        if (int32_t rc = launch_one(ctx, p, w->type)) return rc;
    }
    return TLC_OK;
}
