// Matrix products with the WEIGHT rows on the M side of the MMA (tcgen05 + TMEM):
//
//   y[m, n] = sum_k W[n, k] . x[m, k]        W in Q4_0 / Q8_0 blocks or f16; or x . B with B [K, N]
//
// for the activation counts where tlc_gemm_kernel.cuh, which puts 128 activation rows on the M
// side, either pads most of its tile (up to 100 rows) or has too few tiles for 148 SMs.
// A tile is 128 weight rows x bn activation rows (bn any multiple of 16 up to 256).  Two ways to fill 148 SMs:
//   cluster  each tile's K steps are shared out over the ks CTAs of a thread-block cluster, which add their
//            sums through distributed shared memory: small weights, where a call is a few microseconds;
//   stream   the K steps of all tiles, laid end to end, are dealt out evenly to one persistent CTA per SM:
//            large weights, where a last wave would cost more than the hand-over.  A tile whose steps lie
//            with several CTAs is finished by the one that has its last step; the others leave their f32
//            sums in global memory (L2) and raise a flag.  A CTA goes through its steps from the top
//            down: what others wait for comes first, and a CTA waits only for CTAs of lower index, which
//            the hardware starts before it.
//
// What bounds it: up to about 100 activation rows the weight bytes (HBM), or, where the weight is
// small, the chain fetch -> unpack -> MMA -> reduce of one CTA; beyond, the unpacking and the MMAs.
// The unpacked weights never touch shared memory: a thread owns one weight row, turns the row's
// quants into f16 pairs in registers and stores them to TENSOR MEMORY (tcgen05.st), from where
// the MMA takes its A operand.  Shared memory carries the raw blocks (0.56 or 1.06 bytes per
// weight) and the activations only; with the f16 weight tile in shared memory its write and the
// MMA's read of it alone would take more than the 128 bytes a clock that an SM has.
//
// Warps:  0  x producer: TMA boxes of 64 columns x bn rows (128-byte swizzle), after the
//            dependency wait (x comes from the previous kernel)
//         1  producer of quantized weights, started before that wait (weights are never written by a kernel): one
//            TMA box of eight slabs x one tile.  (Dense operands come with the activations, by warp 0 behind the
//            wait: matmul's may be what the previous kernel computed.)  The box takes 16 bytes of the next tile along, so
//            that slabs lie off a multiple of 128 bytes apart and the eight lanes of a 16-byte shared
//            load, which own rows of four slabs, meet different banks.
//         2  tensor memory and MMA issue
//         4-7   epilogue, while the MMAs of the next tile run (two accumulators, up to 128 activation rows)
//         8-23  four groups of four: unpack K step i in group i % 4
#include <cuda.h>

#include <cstring>

#include "tlc_gemm_kernel.cuh"
#include "tlc_gemm_wt.h"

using namespace tlc_gemm;

namespace {

constexpr int kGroups = 4;                      // unpacking groups of four warps
constexpr int kChunk = 32;                     // activation rows per round of the epilogue
constexpr int kMaxRaw = 12, kMaxX = 8, kMaxA = 7;
constexpr int kHeader = 1024;
constexpr int kStagePitch = 160;  // f32 per activation row of the epilogue staging (see fpos)
constexpr int kSumPitch = 144;    // ... of a CTA's sums for the cluster: two rows apart meet all banks (see sum8)

struct WtOut {
    const uint8_t *w;
    size_t slab_pitch;
    int n;      // weight rows (outputs)
    int tiles;  // 128-row tiles (64-row tiles of each weight for the SiLU.mul pair)
    __half *y;
    long long row_stride, pos_stride;
    int head_dim;  // > 0: interleaved RoPE
};

struct WtMaps {
    CUtensorMap m[3];
};

struct WtParams {
    WtOut out[3];
    const uint8_t *w2;  // up weight of the SiLU.mul pair (out[0] is the gate), or null
    int k_tiles;        // quantized weights: tiles per slab
    int steps;          // K steps of a tile
    long long total_steps;
    int grid;
    int ks;             // cluster form: CTAs per tile; 0: stream form
    int own_gather;     // cluster form: the sums' place is not in the rings
    int m, bn, tm;      // activation rows, of a tile, tiles of them
    int raw_stages, x_stages, a_stages, acc_stages;
    int tmem_cols, a_col0, a_col_a;  // columns of an accumulator; first column of the A stages
    float *partial;     // [CTA][bn][128]: the sums of a tile's part (a CTA leaves at most one)
    int *flags;         // [CTA]: its part is there; zero between launches
    const __half *bias, *residual;
    int pos_offset;
    const int *positions;
    int max_pos;
    float rope_base;
    int vec_ok;
    tlc_dev_status *status;
    uint64_t wait_ns;
};

template <int SRC> struct Src;
template <> struct Src<kWtQ4> { static constexpr bool DQ = true; static constexpr int KSTEP = 128, TILE = 1152, TPS = 1; };
template <> struct Src<kWtQ8> { static constexpr bool DQ = true; static constexpr int KSTEP = 128, TILE = 1088, TPS = 2; };
template <> struct Src<kWtF16> { static constexpr bool DQ = false; static constexpr int KSTEP = 64, TILE = 0, TPS = 0; };
template <> struct Src<kWtF16T> { static constexpr bool DQ = false; static constexpr int KSTEP = 64, TILE = 0, TPS = 0; };
// A staged tile of eight slabs: rows of TILE + 16 bytes; the second four slabs (another box when they are the
// up rows of a SiLU.mul pair) start on a multiple of 128 bytes.
template <int SRC> constexpr int slab_bytes() { return Src<SRC>::TILE + 16; }
template <int SRC> constexpr int box_bytes() { return Src<SRC>::DQ ? 8 * slab_bytes<SRC>() + 128 - 8 * slab_bytes<SRC>() % 128 : 0; }
template <int SRC> constexpr int raw_stage_bytes() { return Src<SRC>::TPS * box_bytes<SRC>(); }
constexpr int kPairPad = 64;
template <int SRC> constexpr int threads_of() { return Src<SRC>::DQ ? 256 + 128 * kGroups : 256; }
constexpr int kATile = 128 * 64 * 2;  // f16 weights: one K step of the A operand in shared memory

// Position of weight row n (0..127) in a row of the epilogue staging: the lanes of a warp that
// unpacked quantized weights hold rows of eight slabs, 16 apart; 20 apart they meet 32 banks.
__device__ __forceinline__ int fpos(int n) { return n + ((n >> 4) << 2); }

// 16 consecutive tensor-memory columns of this thread's lane.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ bool mbar_test_wait(uint64_t *bar, uint32_t parity) {  // (does not suspend)
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for another CTA's flag.
__device__ __forceinline__ bool flag_wait(const int *flag, volatile int *abort_flag, tlc_dev_status *status, uint64_t wait_ns) {
    uint64_t t0 = 0;
    for (int spin = 1;; spin++) {
        int v;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (v) return true;
        if ((spin & 31) == 0) {
            const uint64_t now = tlc_globaltimer_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 >= (*abort_flag ? 20000ull : wait_ns)) break;
        }
    }
    *abort_flag = 1;
    if (atomicCAS(&status->code, 0, 2) == 0) status->where = 29;
    return false;
}
// Weight row (slab of the tile, row of the slab) of lane `lane` of tensor-memory quarter q, quantized weights.
__device__ __forceinline__ int lane_slab(int lane) { return (lane >> 1) & 7; }
__device__ __forceinline__ int lane_row(int q, int lane) { return 4 * q + 2 * (lane >> 4) + (lane & 1); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t u32(const __half2 &h) { return *reinterpret_cast<const uint32_t *>(&h); }
__device__ __forceinline__ __half2 h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }

// One Q4_0 block: its four quant words and its scale -> 32 f16 weights in K order (16 pairs).
// f16((q - 8) * d) with one rounding, as the reference's loader computes it: a nibble in the low
// mantissa bits of 1024.0 is 1024 + q, in the next four bits 1024 + 16 q; both minus their offset are
// exact, the product with d rounds once.
__device__ __forceinline__ void unpack_q4(const uint32_t (&q)[4], __half2 d2, uint32_t (&o)[16]) {
    const __half2 m1032 = __float2half2_rn(-1032.f), m72 = __float2half2_rn(-72.f), r16 = __float2half2_rn(0.0625f);
#pragma unroll
    for (int t = 0; t < 4; t++) {
        const uint32_t p0 = __byte_perm(q[t], 0, 0x4140), p1 = __byte_perm(q[t], 0, 0x4342);
        o[2 * t] = u32(__hmul2(__hadd2(h2((p0 & 0x000F000Fu) | 0x64006400u), m1032), d2));
        o[2 * t + 1] = u32(__hmul2(__hadd2(h2((p1 & 0x000F000Fu) | 0x64006400u), m1032), d2));
        o[8 + 2 * t] = u32(__hmul2(__hfma2(h2((p0 & 0x00F000F0u) | 0x64006400u), r16, m72), d2));
        o[8 + 2 * t + 1] = u32(__hmul2(__hfma2(h2((p1 & 0x00F000F0u) | 0x64006400u), r16, m72), d2));
    }
}
// One Q8_0 block (eight words).
__device__ __forceinline__ void unpack_q8(const uint32_t (&q)[8], __half2 d2, uint32_t (&o)[16]) {
    const __half2 m1152 = __float2half2_rn(-1152.f);
#pragma unroll
    for (int w = 0; w < 8; w++) {
        const uint32_t u = q[w] ^ 0x80808080u;
        o[2 * w] = u32(__hmul2(__hadd2(bytes_to_half2(u, 0x4140), m1152), d2));
        o[2 * w + 1] = u32(__hmul2(__hadd2(bytes_to_half2(u, 0x4342), m1152), d2));
    }
}

// Place in a ring of `n` stages and the parity its next wait is for.  (Counted, not divided: the loops
// below are serial chains of one warp each, and an integer division costs as much as the hand-over.)
struct Ring {
    int s = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void next(int n) {
        if (++s == n) {
            s = 0;
            ph ^= 1u;
        }
    }
    __device__ __forceinline__ void skip(int n) {  // kGroups places on
        s += kGroups;
        while (s >= n) {
            s -= n;
            ph ^= 1u;
        }
    }
};

// One activation row, eight consecutive outputs n .. n + 7 from their f32 sums (`u`: the up projection's): f16
// rounding, then SiLU.mul / RoPE / bias / residual as the launch asks.
__device__ __forceinline__ void store_item(const WtParams &p, const WtOut &out, bool pair, const float (&v)[8], const float (&u)[8],
                                           int row, int n) {
    const int pos = p.positions ? p.positions[row] : p.pos_offset + row;
    if (out.pos_stride != 0 && p.max_pos > 0 && (pos < 0 || pos >= p.max_pos)) {
        if (atomicCAS(&p.status->code, 0, TLC_DEV_INDEX) == 0) p.status->where = 303;
        return;
    }
    __align__(16) __half h[8];
#pragma unroll
    for (int e = 0; e < 8; e++) h[e] = __float2half_rn(v[e]);
    if (pair) {
        // s = sigmoid(g) (f32, RNE); a = g*s; act = a*u: three f16 roundings as in
        // debug/chat_demo_with_kvcache.tl:26-41
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const __half sg = __float2half_rn(1.0f / (1.0f + expf(-__half2float(h[e]))));
            h[e] = __hmul(__hmul(h[e], sg), __float2half_rn(u[e]));
        }
    } else if (out.head_dim > 0) {
        // interleaved RoPE on the f16-rounded projection (rope_f16, shaders/unified.metal:2355-2417)
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
            const int i2 = ((n + e) % out.head_dim) & ~1;
            const float freq = 1.0f / powf(p.rope_base, (float)i2 / (float)out.head_dim);
            const float theta = (float)(unsigned)pos * freq;
            const float cs = cosf(theta), sn = sinf(theta);
            const float x0 = __half2float(h[e]), x1 = __half2float(h[e + 1]);
            h[e] = __float2half_rn(__fsub_rn(__fmul_rn(x0, cs), __fmul_rn(x1, sn)));
            h[e + 1] = __float2half_rn(__fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, cs)));
        }
    }
    const int left = out.n - n;  // outputs of this item that exist
    if (p.bias) {
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (e < left) h[e] = __hadd(h[e], p.bias[n + e]);
    }
    const bool vec = p.vec_ok && left >= 8;
    if (p.residual) {
        const __half *rr = p.residual + (size_t)row * out.n + n;
        __align__(16) __half rv[8];
        if (vec) *reinterpret_cast<uint4 *>(rv) = *reinterpret_cast<const uint4 *>(rr);
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (e < left) h[e] = __hadd(h[e], vec ? rv[e] : rr[e]);
    }
    __half *y = out.y + (size_t)((long long)row * out.row_stride + (long long)pos * out.pos_stride) + n;
    if (vec) {
        *reinterpret_cast<uint4 *>(y) = *reinterpret_cast<const uint4 *>(h);
    } else {
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (e < left) y[e] = h[e];
    }
}

__device__ __forceinline__ void load8(const float *at, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4 *>(at), b = *reinterpret_cast<const float4 *>(at + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// The cluster's sums of eight consecutive weight rows from n on, added in rank order.  They lie in tensor-memory
// lane order (`at`: this activation row's from rank 0, `part`: f32 from one rank's to the next one's), where
// the lanes of quantized weights hold the rows of a slab in pairs 16 apart.
template <bool DQ>
__device__ __forceinline__ void sum8(const float *at, int part, int ks, int n, float (&v)[8]) {
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = 0.f;
    const float *src = at + (DQ ? ((n & 15) >> 1) * 16 + (n >> 4) * 2 : n);
#pragma unroll 2
    for (int r = 0; r < ks; r++, src += part)
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
            const float2 t = *reinterpret_cast<const float2 *>(src + (DQ ? 8 * e : e));
            v[e] += t.x;
            v[e + 1] += t.y;
        }
}

// A piece of a CTA's work: K steps [k0, k0 + n) of a tile.  A CTA owns the steps [lo, hi) of all
// tiles laid end to end and takes them tile by tile from the top down.
struct Segment {
    int tile, k0, n;
};
__device__ __forceinline__ long long range_lo(const WtParams &p, int g) { return (long long)p.total_steps * g / p.grid; }
__device__ __forceinline__ Segment segment_below(const WtParams &p, long long lo, long long hi) {
    Segment s;
    s.tile = (int)((hi - 1) / p.steps);
    const long long t0 = (long long)s.tile * p.steps;
    s.k0 = (int)((lo > t0 ? lo : t0) - t0);
    s.n = (int)(hi - t0) - s.k0;
    return s;
}

template <int SRC, bool CLUSTER>
__global__ void __launch_bounds__(threads_of<SRC>(), 1)
    gemm_wt_kernel(const __grid_constant__ WtParams p, const __grid_constant__ CUtensorMap x_map,
                   const __grid_constant__ WtMaps w_maps) {
    using S = Src<SRC>;
    constexpr bool DQ = S::DQ;
    constexpr int KSTEP = S::KSTEP;
    constexpr int SLAB = slab_bytes<SRC>();
    constexpr int RAW = raw_stage_bytes<SRC>();

    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *raw_full = reinterpret_cast<uint64_t *>(base), *raw_empty = raw_full + kMaxRaw;
    uint64_t *x_full = raw_empty + kMaxRaw, *x_empty = x_full + kMaxX;
    uint64_t *a_full = x_empty + kMaxX, *a_empty = a_full + kMaxA;
    uint64_t *acc_full = a_empty + kMaxA, *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    uint8_t *rings = base + kHeader;
    const int x_bytes = p.bn * KSTEP * 2;
    const int x_stage = x_bytes + (DQ ? 0 : kATile);  // f16 weights: the A tile lies behind the x tile
    uint8_t *raw = rings + (size_t)p.x_stages * x_stage;
    // stream form: staging of the epilogue; cluster form: the sums of this CTA's activation rows, from every rank
    float *staging = reinterpret_cast<float *>(CLUSTER && !p.own_gather ? rings : raw + (size_t)p.raw_stages * RAW);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const bool pair = p.w2 != nullptr;
    const int g = blockIdx.x;
    // this CTA's steps (never none: see the launcher)
    long long lo, hi;
    int rank = 0;
    if (CLUSTER) {
        const int tile = g / p.ks, per = (p.steps + p.ks - 1) / p.ks;
        rank = g - tile * p.ks;
        lo = (long long)tile * p.steps + rank * per;
        hi = (long long)tile * p.steps + min(p.steps, (rank + 1) * per);
    } else {
        lo = range_lo(p, g);
        hi = range_lo(p, g + 1);
    }

    if (tid == 0) {
        for (int i = 0; i < p.raw_stages; i++) {
            mbar_init(&raw_full[i], 1);
            mbar_init(&raw_empty[i], 4);
        }
        for (int i = 0; i < p.x_stages; i++) {
            mbar_init(&x_full[i], 1);
            mbar_init(&x_empty[i], 1);
        }
        for (int i = 0; i < p.a_stages; i++) {
            mbar_init(&a_full[i], 4);
            mbar_init(&a_empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(p.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // (the peers may write to this CTA's shared memory from here on)
    if (CLUSTER && p.own_gather) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    // tile -> (output, tile of that output's rows, tile of activation rows)
    auto locate = [&](int tile, int &oi, int &tn, int &m0) {
        tn = tile / p.tm;
        m0 = (tile - tn * p.tm) * p.bn;
        oi = 0;
        if (!pair) {
            if (tn >= p.out[0].tiles) { tn -= p.out[0].tiles; oi = 1; }
            if (oi == 1 && tn >= p.out[1].tiles) { tn -= p.out[1].tiles; oi = 2; }
        }
    };

    if (warp == 0) {
        // ------------------------------ activations ------------------------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        const uint32_t el = elect_one();
        Ring rx;
        bool ok = true;
        for (long long h = hi; ok && h > lo;) {
            const Segment sg = segment_below(p, lo, h);
            h -= sg.n;
            int oi, tn, m0;
            locate(sg.tile, oi, tn, m0);
            for (int i = 0; i < sg.n; i++, rx.next(p.x_stages)) {
                const int s = rx.s;
                ok = __all_sync(0xffffffffu, mbar_wait(&x_empty[s], rx.ph ^ 1u, abort_flag, p.status, 21, p.wait_ns));
                if (!ok) break;
                const uint32_t bar = smem_u32(&x_full[s]);
                const uint32_t dst = smem_u32(rings + (size_t)s * x_stage);
                mbar_arrive_expect_tx_el(&x_full[s], (uint32_t)x_stage, el);
                const int k = (sg.k0 + i) * KSTEP;
#pragma unroll
                for (int q = 0; q < KSTEP / 64; q++) tma_load_2d_el(dst + q * (p.bn * 128), &x_map, k + 64 * q, m0, bar, el);
                if (SRC == kWtF16) tma_load_2d_el(dst + x_bytes, &w_maps.m[0], k, tn * 128, bar, el);
                if (SRC == kWtF16T) {
                    tma_load_2d_el(dst + x_bytes, &w_maps.m[0], tn * 128, k, bar, el);
                    tma_load_2d_el(dst + x_bytes + kATile / 2, &w_maps.m[0], tn * 128 + 64, k, bar, el);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------ raw weights ------------------------------
        if constexpr (DQ) {
            const uint32_t el = elect_one();
            Ring rr;
            bool ok = true;
            for (long long h = hi; ok && h > lo;) {
                const Segment sg = segment_below(p, lo, h);
                h -= sg.n;
                int oi, tn, m0;
                locate(sg.tile, oi, tn, m0);
                const void *map = &w_maps.m[oi];
                for (int i = 0; i < sg.n; i++, rr.next(p.raw_stages)) {
                    const int s = rr.s;
                    ok = __all_sync(0xffffffffu, mbar_wait(&raw_empty[s], rr.ph ^ 1u, abort_flag, p.status, 22, p.wait_ns));
                    if (!ok) break;
                    const int kt = (sg.k0 + i) * S::TPS, nt = min(S::TPS, p.k_tiles - kt);
                    const uint32_t bar = smem_u32(&raw_full[s]), dst = smem_u32(raw + (size_t)s * RAW);
                    mbar_arrive_expect_tx_el(&raw_full[s], (uint32_t)(nt * 8 * SLAB), el);
#pragma unroll
                    for (int j = 0; j < S::TPS; j++) {
                        if (j >= nt) break;
                        const int x = (kt + j) * (S::TILE / 8);  // the maps count in 8-byte elements
                        const uint32_t d = dst + j * box_bytes<SRC>();
                        if (pair) {
                            tma_load_2d_el(d, &w_maps.m[0], x, tn * 4, bar, el);
                            tma_load_2d_el(d + 4 * SLAB + kPairPad, &w_maps.m[1], x, tn * 4, bar, el);
                        } else {
                            tma_load_2d_el(d, map, x, tn * 8, bar, el);
                        }
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // ------------------------------ MMA ------------------------------
        const uint32_t idesc = idesc_for(p.bn) | (SRC == kWtF16T ? 1u << 15 : 0u);
        // K-major operands (desc_at) and, for the dense [K, N] matrix, an N-major one: TMA boxes of 64 n x 64 k,
        // eight k 1024 bytes apart (the stride offset), the next 64 n the next box (the leading offset).
        constexpr uint32_t MN = (uint32_t)((64 * 128) >> 4) << 16;
        const uint32_t x0 = (smem_u32(rings) & 0x3FFFF) >> 4, x_step = (uint32_t)x_stage >> 4;
        const uint32_t half = (uint32_t)(p.bn * 128) >> 4, a_off = (uint32_t)x_bytes >> 4;
        const uint32_t el = elect_one();
        Ring rx, ra, rc;
        // The next step's barriers are looked at while this step's MMAs are issued: a wait costs about
        // 110 clocks even when there is nothing to wait for.
        bool px = false, pa = false;
        for (long long h = hi; h > lo;) {
            const Segment sg = segment_below(p, lo, h);
            h -= sg.n;
            bool ready = mbar_wait(&acc_empty[rc.s], rc.ph ^ 1u, abort_flag, p.status, 28, p.wait_ns);
            const uint32_t acc_at = tmem + rc.s * p.a_col0;
            uint32_t acc = 0;
            for (int i = 0; i < sg.n; i++) {
                if (!px) ready = mbar_wait(&x_full[rx.s], rx.ph, abort_flag, p.status, 23, p.wait_ns) && ready;
                if (DQ && !pa) ready = mbar_wait(&a_full[ra.s], ra.ph, abort_flag, p.status, 24, p.wait_ns) && ready;
                ready = __all_sync(0xffffffffu, ready);
                tc_fence_after();
                const uint32_t xa = x0 + rx.s * x_step, ta = tmem + p.a_col_a + ra.s * 64;
                const int xs = rx.s, as = ra.s;
                rx.next(p.x_stages);
                ra.next(p.a_stages);
                px = mbar_test_wait(&x_full[rx.s], rx.ph);
                if (DQ) pa = mbar_test_wait(&a_full[ra.s], ra.ph);
                if (ready) {
#pragma unroll
                    for (int k16 = 0; k16 < KSTEP / 16; k16++) {
                        const uint64_t bdesc = desc_at(xa + (k16 >> 2) * half + (k16 & 3) * 2);
                        if (DQ)
                            umma_f16_ts(acc_at, ta + k16 * 8, bdesc, idesc, acc, el);
                        else if (SRC == kWtF16)
                            umma_f16(acc_at, desc_at(xa + a_off + k16 * 2), bdesc, idesc, acc, el);
                        else
                            umma_f16(acc_at, (desc_at(xa + a_off + k16 * 128) & ~(uint64_t)(1u << 16)) | MN, bdesc, idesc, acc, el);
                        acc = 1;
                    }
                }
                umma_commit(&x_empty[xs], el);
                if (DQ) umma_commit(&a_empty[as], el);
            }
            umma_commit(&acc_full[rc.s], el);
            rc.next(p.acc_stages);
        }
        __syncwarp();
    } else if (warp >= 8) {
        if constexpr (DQ) {
            // ------------------------------ unpack ------------------------------
            const int grp = (warp - 8) >> 2, q = warp & 3;
            const uint32_t tlane = tmem + ((uint32_t)(32 * q) << 16);
            // weight row of this lane (tensor-memory lane 32 q + lane): slab, row of the slab
            const int slab = lane_slab(lane), r16 = lane_row(q, lane);
            const uint32_t sbase = (uint32_t)(slab * SLAB + (pair ? (slab >> 2) * kPairPad : 0));
            const uint32_t qoff = sbase + (uint32_t)((r16 >> 3) * 512 + (r16 & 7) * 64);
            const uint32_t soff = sbase + 1024u + (uint32_t)(r16 * (SRC == kWtQ4 ? 8 : 4));
            Ring rr, ra;
            for (int i = 0; i < grp; i++) {
                rr.next(p.raw_stages);
                ra.next(p.a_stages);
            }
            // K steps of the CTA in the order they are produced; `k`: step of its tile (Q8_0: the last may be half)
            Segment sg = segment_below(p, lo, hi);
            long long h = hi;
            int at = 0;
            auto forward = [&](int by) {
                at += by;
                while (at >= sg.n && h > lo) {
                    at -= sg.n;
                    h -= sg.n;
                    if (h > lo) sg = segment_below(p, lo, h);
                }
            };
            forward(grp);
            for (; h > lo; forward(kGroups), rr.skip(p.raw_stages), ra.skip(p.a_stages)) {
                const int s = rr.s, as = ra.s;
                mbar_wait(&raw_full[s], rr.ph, abort_flag, p.status, 25, p.wait_ns);
                __syncwarp();  // the lanes leave a wait one by one; what follows is for a whole warp
                const uint32_t rb = smem_u32(raw + (size_t)s * RAW);
                uint4 v[4 * S::TPS];
                uint32_t sc[2];
#pragma unroll
                for (int j = 0; j < S::TPS; j++)
#pragma unroll
                    for (int t = 0; t < 4; t++) v[4 * j + t] = lds128(rb + qoff + j * box_bytes<SRC>() + 16 * t);
                if (SRC == kWtQ4) {
                    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(sc[0]), "=r"(sc[1]) : "r"(rb + soff));
                } else {
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sc[0]) : "r"(rb + soff));
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sc[1]) : "r"(rb + soff + box_bytes<SRC>()));
                    // a last step of one tile: the second one was not copied; its scales are zero
                    if ((sg.k0 + at) * S::TPS + 1 >= p.k_tiles) sc[1] = 0;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[s]);
                mbar_wait(&a_empty[as], ra.ph ^ 1u, abort_flag, p.status, 26, p.wait_ns);
                __syncwarp();
                tc_fence_after();
                const uint32_t ta = tlane + p.a_col_a + as * 64;
#pragma unroll
                for (int j = 0; j < 4; j++) {  // the four blocks of the step
                    const __half2 d2 = __half2half2(__ushort_as_half((unsigned short)(j & 1 ? sc[j >> 1] >> 16 : sc[j >> 1] & 0xFFFFu)));
                    uint32_t o[16];
                    auto comp = [](const uint4 &u, int c) { return c == 0 ? u.x : c == 1 ? u.y : c == 2 ? u.z : u.w; };
                    if (SRC == kWtQ4) {
                        const uint32_t w[4] = {comp(v[0], j), comp(v[1], j), comp(v[2], j), comp(v[3], j)};
                        unpack_q4(w, d2, o);
                    } else {
                        uint32_t w[8];
#pragma unroll
                        for (int t = 0; t < 4; t++) {
                            w[2 * t] = comp(v[(S::TPS - 1) * 4 * (j >> 1) + t], 2 * (j & 1));
                            w[2 * t + 1] = comp(v[(S::TPS - 1) * 4 * (j >> 1) + t], 2 * (j & 1) + 1);
                        }
                        unpack_q8(w, d2, o);
                    }
                    tmem_st16(ta + 16 * j, o);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[as]);
            }
        }
    } else if (warp >= 4) {
        // ------------------------------ epilogue ------------------------------
        asm volatile("griddepcontrol.wait;" ::: "memory");  // residual, positions, the outputs and the partial sums
        const int q = warp & 3, et = tid - 128;
        const int n_local = DQ ? lane_slab(lane) * 16 + lane_row(q, lane) : 32 * q + lane;
        const size_t slot = (size_t)p.bn * 128;  // f32 sums of a part of a tile: [activation row][tensor-memory lane]
        Ring rc;
        for (long long h = hi; h > lo;) {
            const Segment sg = segment_below(p, lo, h);
            h -= sg.n;
            int oi, tn, m0;
            locate(sg.tile, oi, tn, m0);
            const WtOut &out = p.out[oi];
            mbar_wait(&acc_full[rc.s], rc.ph, abort_flag, p.status, 27, p.wait_ns);
            __syncwarp();
            tc_fence_after();
            const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + rc.s * p.a_col0;
            if (CLUSTER) break;  // the one tile of this CTA
            if (sg.k0 + sg.n < p.steps) {
                // The tile's last steps are with the next CTAs: leave the sums for the one that has the very last.
                float *dst = p.partial + (size_t)g * slot + 32 * q + lane;
                for (int c0 = 0; c0 < p.bn; c0 += 16) {
                    uint32_t r[16];
                    tmem_ld16(taddr + c0, r);
#pragma unroll
                    for (int e = 0; e < 16; e++) __stcg(dst + (size_t)(c0 + e) * 128, __uint_as_float(r[e]));
                }
                tc_fence_before();
                __threadfence();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[rc.s]);
                rc.next(p.acc_stages);
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (et == 0) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p.flags + g), "r"(1) : "memory");
                continue;
            }
            // How many CTAs below hold earlier steps of the tile, and are they done?
            int parts = 0;
            if (sg.k0 > 0) {
                const long long t0 = (long long)sg.tile * p.steps;
                int gg = g - 1;
                while (range_lo(p, gg) > t0) gg--;
                parts = g - gg;
                for (int pt = et; pt < parts; pt += 128) {
                    flag_wait(p.flags + g - 1 - pt, abort_flag, p.status, p.wait_ns);
                    p.flags[g - 1 - pt] = 0;
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                __threadfence();
            }
            const float *src = p.partial + (size_t)(g - 1) * slot + 32 * q + lane;
            const int rows = min(p.bn, p.m - m0), groups = pair ? 8 : 16, n_base = tn * (pair ? 64 : 128);
            for (int c0 = 0; c0 < p.bn; c0 += kChunk) {
                const int cols = min(kChunk, p.bn - c0);
#pragma unroll
                for (int h16 = 0; h16 < kChunk; h16 += 16) {
                    if (h16 >= cols) break;
                    uint32_t r[16];
                    __syncwarp();
                    tmem_ld16(taddr + c0 + h16, r);
                    float *dst = staging + (size_t)h16 * kStagePitch + fpos(n_local);
                    for (int pt = 0; pt < parts; pt += 2) {  // two parts' loads in flight
                        const float *sp = src - (size_t)pt * slot + (size_t)(c0 + h16) * 128;
                        const bool two = pt + 1 < parts;
                        float t[16], t2[16];
#pragma unroll
                        for (int e = 0; e < 16; e++) t[e] = __ldcg(sp + e * 128);
#pragma unroll
                        for (int e = 0; e < 16; e++) t2[e] = two ? __ldcg(sp - slot + e * 128) : 0.f;
#pragma unroll
                        for (int e = 0; e < 16; e++) r[e] = __float_as_uint(__uint_as_float(r[e]) + t[e] + t2[e]);
                    }
#pragma unroll
                    for (int e = 0; e < 16; e++) dst[e * kStagePitch] = __uint_as_float(r[e]);
                }
                if (c0 + kChunk >= p.bn) {  // the accumulator has been read
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[rc.s]);
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
                for (int item = et; item < min(cols, rows - c0) * groups; item += 128) {
                    const int c = pair ? item >> 3 : item >> 4, g8 = (pair ? item & 7 : item & 15) * 8;
                    const int n = n_base + g8;
                    if (n >= out.n) continue;
                    float v[8], u[8];
                    load8(staging + (size_t)c * kStagePitch + fpos(g8), v);
                    if (pair) load8(staging + (size_t)c * kStagePitch + fpos(64 + g8), u);
                    store_item(p, out, pair, v, u, m0 + c0 + c, n);
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
            }
            rc.next(p.acc_stages);
        }
    }
    if (CLUSTER) {
        // The CTAs of the cluster take the activation rows in turn.  Each stores its sums where their owner adds them
        // up: stores need no answer, where loads from the peers took a microsecond and a barrier to let them leave
        // (2048 x 2048, 32 rows: 8.3 -> 7.7 us; 4096 x 4096, 64 rows:
        // 12.3 -> 10.7).  Without a place of their own the sums go over the rings, which the peers have to be done
        // with first.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        __syncwarp();
        if (!p.own_gather) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int tile = g / p.ks;
        int oi, tn, m0;
        locate(tile, oi, tn, m0);
        const WtOut &out = p.out[oi];
        const int rows = min(p.bn, p.m - m0), groups = pair ? 8 : 16, n_base = tn * (pair ? 64 : 128);
        const int part = (p.bn + p.ks - 1) / p.ks * kSumPitch;
        if (warp >= 4 && warp < 8) {
            const int q = warp & 3;
            uint32_t at = smem_u32(staging + rank * part + 32 * q + lane);
            int owner = 0;
            for (int c0 = 0; c0 < rows; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + c0, r);
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    uint32_t ra;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(at), "r"(owner));
                    if (c0 + e < rows) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(ra), "r"(r[e]) : "memory");
                    if (++owner == p.ks) {
                        owner = 0;
                        at += kSumPitch * 4;
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int mine = (rows - rank + p.ks - 1) / p.ks;
        for (int item = tid; item < mine * groups; item += threads_of<SRC>()) {
            const int i = pair ? item >> 3 : item >> 4, g8 = (pair ? item & 7 : item & 15) * 8;
            const int n = n_base + g8;
            if (n >= out.n) continue;
            float v[8], u[8];
            sum8<DQ>(staging + i * kSumPitch, part, p.ks, g8, v);
            if (pair) sum8<DQ>(staging + i * kSumPitch, part, p.ks, 64 + g8, u);
            store_item(p, out, pair, v, u, m0 + i * p.ks + rank, n);
        }
    }
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
    }
}

// Rows of odd lengths or addresses, brought to a pitch TMA can read (a multiple of eight f16).
struct PitchJob {
    const __half *src;
    __half *dst;
    long long rows;
    int cols, pitch;
};
__global__ void __launch_bounds__(256) pitch_rows_kernel(PitchJob a, PitchJob b) {
    tlc_pdl_prologue();
    const PitchJob j = blockIdx.y == 0 ? a : b;
    const int per = j.pitch >> 3;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < j.rows * per; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / per;
        const int c = (int)(i - r * per) * 8;
        __align__(16) __half v[8];
        const __half *s = j.src + r * j.cols + c;
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = c + e < j.cols ? s[e] : __ushort_as_half((unsigned short)0);
        *reinterpret_cast<uint4 *>(j.dst + r * j.pitch + c) = *reinterpret_cast<const uint4 *>(v);
    }
}

struct Plan {
    int bn, tm, grid, ks;
};

template <int SRC> int max_clusters(tlc_ctx *ctx, int ks);

// Activation rows per tile, form and CTAs.  Cost in microseconds.  A K step is bound by the unpacking
// (`unpack`), the MMAs (128 x bn x 16 take bn / 2 clocks, 36 at least) or the bytes that reach the SM (x from L2
// and the raw weights).  Cluster form: whole waves of clusters, each with a start, a fill and a drain.  Stream
// form: the share of one SM once, and the hand-over of the tiles that several CTAs hold.
template <int SRC>
Plan choose_plan(tlc_ctx *ctx, int m, int64_t tiles_n, int steps, double unpack) {
    const double kstep = Src<SRC>::KSTEP, raw_bytes = Src<SRC>::DQ ? raw_stage_bytes<SRC>() : kATile;
    Plan best{16, (m + 15) / 16, 1, 0};
    double best_t = 1e30;
    int last_bn = 0;
    for (int tm = (m + 255) / 256; tm <= (m + 15) / 16; tm++) {
        int bn = ((m + tm - 1) / tm + 15) / 16 * 16;
        if (ctx->gemm_wt_bn) bn = ctx->gemm_wt_bn;
        if (bn == last_bn) continue;
        last_bn = bn;
        const int tmr = (m + bn - 1) / bn;
        const double clk = 1.0 / 1850.0, k16 = kstep / 16;
        const double mma = (k16 * (bn > 72 ? bn * 0.5 : 36.0) + 130.0) * clk, feed = (bn * kstep * 2 + raw_bytes) / 72000.0;
        double step = mma > feed ? mma : feed;
        step = step > unpack ? step : unpack;
        const int64_t tiles = tiles_n * tmr, total = tiles * steps;
        for (int ks = 1; ks <= 8 && ks <= steps; ks++) {
            const int per = (steps + ks - 1) / ks;
            if ((ks - 1) * per >= steps) continue;  // a share would be empty
            if (ctx->gemm_wt_ks == 9) continue;
            if (ctx->gemm_wt_ks && ks != (ctx->gemm_wt_ks < steps ? ctx->gemm_wt_ks : steps)) continue;
            const int64_t fit = max_clusters<SRC>(ctx, ks);
            if (fit < 1) continue;
            const double waves = (double)((tiles + fit - 1) / fit);
            const double t = waves * (per * step + 3.0 + bn * 0.012) + (ks > 1 ? 1.0 + bn * 0.01 : 0.0);
            if (t < best_t) {
                best_t = t;
                best = {bn, tmr, (int)(tiles * ks), ks};
            }
        }
        if (ctx->gemm_wt_ks && ctx->gemm_wt_ks < 9) continue;
        const int64_t grid = ctx->sm_count < total ? ctx->sm_count : total;
        const double share = (double)((total + grid - 1) / grid), parts = share < steps ? (steps + share - 1) / share : 1.0;
        const double t = share * step + 3.5 + bn * 0.012 + 3.0 + parts * bn * 0.03 + (bn > 128 ? share / steps * bn * 0.012 : 0.0);
        if (t < best_t) {
            best_t = t;
            best = {bn, tmr, (int)grid, 0};
        }
    }
    return best;
}

template <int SRC>
int32_t configure(tlc_ctx *ctx) {
    static bool configured[64] = {};
    if (configured[ctx->device & 63]) return TLC_OK;
    const void *fns[2] = {(const void *)gemm_wt_kernel<SRC, true>, (const void *)gemm_wt_kernel<SRC, false>};
    for (const void *fn : fns) {
        TLC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ctx->prop.sharedMemPerBlockOptin));
        TLC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    }
    configured[ctx->device & 63] = true;
    return TLC_OK;
}

// Clusters of ks CTAs that the device holds at once (asked once).
template <int SRC>
int max_clusters(tlc_ctx *ctx, int ks) {
    if (ks == 1) return ctx->sm_count;
    static int known[64][9];
    int &n = known[ctx->device & 63][ks];
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)ks);
        cfg.blockDim = dim3(threads_of<SRC>());
        cfg.dynamicSmemBytes = 200 * 1024;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)ks;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int got = 0;
        if (configure<SRC>(ctx) || cudaOccupancyMaxActiveClusters(&got, gemm_wt_kernel<SRC, true>, &cfg) != cudaSuccess || got < 1) {
            cudaGetLastError();
            got = -1;
        }
        n = got;
    }
    return n;
}

template <int SRC>
int32_t launch(tlc_ctx *ctx, WtParams &p, int tiles_n, const Plan &plan, const CUtensorMap &x_map, const WtMaps &w_maps) {
    using S = Src<SRC>;
    p.bn = plan.bn;
    p.tm = plan.tm;
    p.grid = plan.grid;
    p.ks = plan.ks;
    p.total_steps = (long long)tiles_n * p.tm * p.steps;
    p.partial = ctx->wt_partial;
    p.flags = ctx->wt_flags;
    const size_t x_stage = (size_t)p.bn * S::KSTEP * 2 + (S::DQ ? 0 : kATile), RAW = raw_stage_bytes<SRC>();
    // The cluster's sums get a place of their own while it costs the rings little (up to 64 activation rows).
    const size_t sums = p.ks ? (size_t)p.ks * ((p.bn + p.ks - 1) / p.ks) * kSumPitch * sizeof(float) : 0;
    p.own_gather = p.ks && sums <= 40 * 1024;
    const size_t stage = p.own_gather ? sums : p.ks ? 0 : (size_t)kChunk * kStagePitch * sizeof(float), budget = (size_t)224 * 1024 - kHeader - 1024 - stage;
    int xs = (int)((S::DQ ? budget / 2 : budget) / x_stage);
    xs = xs < 2 ? 2 : xs > kMaxX ? kMaxX : xs;
    // A raw stage always returns to the same unpacking group (the ring is a multiple of the groups): a
    // group's wait then tells its own step from the one before it on that stage.  With any other
    // length a group that runs ahead can wait on a stage whose load before last has landed and whose last
    // one has not -- loads may land out of order -- and the phase bit cannot tell the two apart.
    int rs = 0;
    if constexpr (S::DQ) {
        rs = (int)((budget - xs * x_stage) / RAW) / kGroups * kGroups;
        rs = rs < kGroups ? kGroups : rs > kMaxRaw ? kMaxRaw : rs;
    }
    p.x_stages = xs;
    p.raw_stages = rs;
    p.a_col0 = (p.bn + 31) / 32 * 32;
    p.acc_stages = p.a_col0 <= 128 ? 2 : 1;
    p.a_col_a = p.acc_stages * p.a_col0;
    // (for the same reason no shorter than the groups are many: a stage's MMAs of two rounds ago are done
    // before its group can come back to it)
    p.a_stages = !S::DQ ? 0 : (512 - p.a_col_a) / 64 < kMaxA ? (512 - p.a_col_a) / 64 : kMaxA;
    const int cols = p.a_col_a + 64 * p.a_stages;
    p.tmem_cols = 32;
    while (p.tmem_cols < cols) p.tmem_cols *= 2;
    size_t smem = xs * x_stage + rs * RAW;
    smem += stage;
    if (p.ks && !p.own_gather && smem < sums) smem = sums;
    smem += kHeader + 1024;
    if (int32_t rc = configure<SRC>(ctx)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.grid);
    cfg.blockDim = dim3(threads_of<SRC>());
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (p.ks > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)p.ks;
        attr[na].val.clusterDim.y = 1;
        attr[na++].val.clusterDim.z = 1;
    }
    if (ctx->use_pdl && ctx->pdl_small) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t le = p.ks ? cudaLaunchKernelEx(&cfg, gemm_wt_kernel<SRC, true>, p, x_map, w_maps)
                                : cudaLaunchKernelEx(&cfg, gemm_wt_kernel<SRC, false>, p, x_map, w_maps);
    if (le != cudaSuccess) {
        cudaGetLastError();
        return tlc_fail(TLC_ERR_CUDA, "gemm launch failed: %s", cudaGetErrorString(le));
    }
    TLC_CHECK_LAUNCH(ctx);
    return TLC_OK;
}

// Tensor map of a weight's tiles: one row per 16-row slab, in 8-byte elements; boxes of `rows` slabs x one tile
// and the 16 bytes behind it.
bool encode_tile_map(CUtensorMap *map, const tlc_qtensor *w, int box_bytes, int rows) {
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, CU_TENSOR_MAP_SWIZZLE_NONE, w->data, w->slab_pitch / 8,
                      (uint64_t)((w->n_rows + 15) / 16), w->slab_pitch, (uint32_t)box_bytes / 8, (uint32_t)rows);
}

int32_t map_failed() { return tlc_fail(TLC_ERR_CUDA, "gemm: no tensor map for these activations"); }

}  // namespace

int32_t tlc_launch_gemm_wt(tlc_ctx *ctx, const tlc_gemv_args &a) {
    const tlc_qtensor *w0 = a.outs[0].w;
    const bool q4 = w0->type == TLC_TYPE_Q4_0, pair = a.epilogue == TLC_EPI_SWIGLU;
    const __half *x = static_cast<const __half *>(a.x);
    TLC_REQUIRE(((uintptr_t)x & 15) == 0, TLC_ERR_INVALID_OPERATION, "gemm: activations must be 16-byte aligned");
    WtParams p{};
    p.m = a.m;
    p.k_tiles = (int)w0->k_tiles;
    p.steps = q4 ? p.k_tiles : (p.k_tiles + 1) / 2;
    p.vec_ok = 1;
    int tiles = 0;
    for (int i = 0; i < (pair ? 1 : a.n_out); i++) {
        const tlc_qtensor *w = a.outs[i].w;
        WtOut &o = p.out[i];
        o.w = static_cast<const uint8_t *>(w->data);
        o.slab_pitch = w->slab_pitch;
        o.n = (int)w->n_rows;
        o.tiles = pair ? (o.n + 63) / 64 : (o.n + 127) / 128;
        o.y = static_cast<__half *>(a.outs[i].y);
        o.row_stride = a.outs[i].row_stride >= 0 ? a.outs[i].row_stride : (long long)w->n_rows;
        o.pos_stride = a.outs[i].pos_stride;
        o.head_dim = a.outs[i].rope_heads > 0 ? (int)(w->n_rows / a.outs[i].rope_heads) : 0;
        if (((o.row_stride | o.pos_stride) & 7) != 0 || ((uintptr_t)o.y & 15) != 0) p.vec_ok = 0;
        tiles += o.tiles;
    }
    if (pair) {
        TLC_REQUIRE(a.outs[1].w->slab_pitch == w0->slab_pitch, TLC_ERR_SHAPE_MISMATCH,
                    "gate and up projections must have the same layout");
        p.w2 = static_cast<const uint8_t *>(a.outs[1].w->data);
    }
    p.bias = a.epilogue == TLC_EPI_STORE ? static_cast<const __half *>(a.bias) : nullptr;
    p.residual = a.epilogue == TLC_EPI_RESIDUAL ? static_cast<const __half *>(a.residual) : nullptr;
    if (p.residual && (((uintptr_t)p.residual & 15) != 0 || (p.out[0].n & 7) != 0)) p.vec_ok = 0;
    p.pos_offset = a.pos_offset;
    p.positions = a.positions;
    p.max_pos = a.max_pos;
    p.rope_base = (float)a.rope_base;
    p.status = ctx->dev_status;
    p.wait_ns = ctx->wait_ns;
    // 0.42 us a K step is what the unpacking takes with all groups busy, 0.5 with the hand-overs of a short share (at 0.3
    // the plans had too many small tiles: 11008 x 4096, 128 rows 30.3 us, now 23.3; 2048 x 5632, 512 rows 25.7, now 19.0)
    const Plan plan = q4 ? choose_plan<kWtQ4>(ctx, a.m, tiles, p.steps, 0.5) : choose_plan<kWtQ8>(ctx, a.m, tiles, p.steps, 0.5);
    CUtensorMap x_map;
    WtMaps w_maps;
    memset(&w_maps, 0, sizeof w_maps);
    for (int i = 0; i < a.n_out; i++)
        if (!encode_tile_map(&w_maps.m[i], a.outs[i].w, q4 ? slab_bytes<kWtQ4>() : slab_bytes<kWtQ8>(), pair ? 4 : 8)) return map_failed();
    if (!encode_f16_map(&x_map, x, (uint64_t)w0->n_cols, (uint64_t)a.m, (uint64_t)w0->n_cols * 2, 64, (uint32_t)plan.bn)) return map_failed();
    return q4 ? launch<kWtQ4>(ctx, p, tiles, plan, x_map, w_maps) : launch<kWtQ8>(ctx, p, tiles, plan, x_map, w_maps);
}

// Dense f16 operands.  `w`: [n, k] rows of w_pitch bytes, or (k_major false) [k, n].
static int32_t dense(tlc_ctx *ctx, const void *w, size_t w_pitch, bool k_major, int n, int k, const void *x, int m, void *y,
                     const void *bias, const void *residual) {
    // TMA wants 16-byte aligned addresses and row pitches; anything else is copied to such a pitch first.
    const int kp = (k + 7) & ~7, np = (n + 7) & ~7;
    const bool px = k != kp || ((uintptr_t)x & 15) != 0;
    const bool pw = k_major ? (w_pitch & 15) != 0 || ((uintptr_t)w & 15) != 0 : n != np || ((uintptr_t)w & 15) != 0;
    if (px || pw) {
        const size_t xb = px ? ((size_t)m * kp * 2 + 255) & ~(size_t)255 : 0;
        const size_t wb = pw ? (k_major ? (size_t)n * kp : (size_t)k * np) * 2 : 0;
        if (int32_t rc = tlc_scratch_reserve(ctx, xb + wb)) return rc;
        __half *sx = static_cast<__half *>(ctx->scratch), *sw = reinterpret_cast<__half *>(static_cast<uint8_t *>(ctx->scratch) + xb);
        const PitchJob jx{static_cast<const __half *>(x), sx, m, k, kp};
        const PitchJob jw{static_cast<const __half *>(w), sw, k_major ? n : k, k_major ? k : n, k_major ? kp : np};
        TLC_REQUIRE(!pw || !k_major || w_pitch == (size_t)k * 2, TLC_ERR_INVALID_OPERATION, "gemm: weight rows are not contiguous");
        const PitchJob &j0 = px ? jx : jw;
        const long long items = j0.rows * (j0.pitch >> 3), items2 = px && pw ? jw.rows * (jw.pitch >> 3) : 0;
        long long blocks = ((items > items2 ? items : items2) + 255) / 256;
        if (blocks > 16LL * ctx->sm_count) blocks = 16LL * ctx->sm_count;
        const cudaError_t le = tlc_launch_pdl(ctx, pitch_rows_kernel, dim3((unsigned)blocks, px && pw ? 2 : 1), dim3(256), 0, j0, jw);
        if (le != cudaSuccess) {
            cudaGetLastError();
            return tlc_fail(TLC_ERR_CUDA, "gemm: row copy failed: %s", cudaGetErrorString(le));
        }
        TLC_CHECK_LAUNCH(ctx);
        if (px) x = sx;
        if (pw) {
            w = sw;
            w_pitch = (size_t)kp * 2;
        }
    }
    WtParams p{};
    p.m = m;
    p.steps = (k + 63) / 64;
    WtOut &o = p.out[0];
    o.n = n;
    o.tiles = (n + 127) / 128;
    o.y = static_cast<__half *>(y);
    o.row_stride = n;
    p.bias = static_cast<const __half *>(bias);
    p.residual = static_cast<const __half *>(residual);
    p.vec_ok = (n & 7) == 0 && ((uintptr_t)y & 15) == 0 && ((uintptr_t)residual & 15) == 0;
    p.status = ctx->dev_status;
    p.wait_ns = ctx->wait_ns;
    const Plan plan = k_major ? choose_plan<kWtF16>(ctx, m, o.tiles, p.steps, 0.0) : choose_plan<kWtF16T>(ctx, m, o.tiles, p.steps, 0.0);
    CUtensorMap x_map;
    WtMaps w_maps;
    memset(&w_maps, 0, sizeof w_maps);
    const uint64_t x_pitch = (uint64_t)kp * 2;
    if (!encode_f16_map(&x_map, x, (uint64_t)k, (uint64_t)m, x_pitch, 64, (uint32_t)plan.bn)) return map_failed();
    if (k_major) {
        if (!encode_f16_map(&w_maps.m[0], w, (uint64_t)k, (uint64_t)n, w_pitch, 64, 128)) return map_failed();
        return launch<kWtF16>(ctx, p, o.tiles, plan, x_map, w_maps);
    }
    if (!encode_f16_map(&w_maps.m[0], w, (uint64_t)n, (uint64_t)k, (uint64_t)np * 2, 64, 64)) return map_failed();
    return launch<kWtF16T>(ctx, p, o.tiles, plan, x_map, w_maps);
}

int32_t tlc_launch_gemm_f16(tlc_ctx *ctx, const void *w, size_t w_pitch, int n, int k, const void *x, int m, void *y,
                            const void *bias, const void *residual) {
    return dense(ctx, w, w_pitch, true, n, k, x, m, y, bias, residual);
}
int32_t tlc_launch_matmul_f16(tlc_ctx *ctx, const void *a, const void *b, void *c, int m, int k, int n) {
    return dense(ctx, b, 0, false, n, k, a, m, c, nullptr, nullptr);
}
