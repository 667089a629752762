// Prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// One CTA owns 128 (query, head) rows that share a KV head -- the G query heads of the group times
// 128/G query positions -- and walks the keys in tiles of 64; two CTAs share an SM, so that one's
// matrix products run under the other's softmax.
//   S = Q.K^T    both operands in shared memory (TMA, 128-byte swizzle), f32 in tensor memory
//   softmax      one row per thread, so that no statistic crosses a lane: tcgen05.ld of the row's 64
//                scores, the two f16 roundings of the reference (einsum output, then the f16 multiply by
//                the scale), online maximum and sum in f32, P rounded to f16 as the reference stores it
//   O += P.V     P from tensor memory (over the scores it was made from), V as it lies in the cache:
//                [key][d] is the N-major form of the operand
// (einsum_ihd_jhd_ihj_f16, apply_attention_mask_f16, softmax_f16 and einsum_ihj_jhd_ihd_f16 of
// shaders/unified.metal:2524-2683, :4474-4488, :2057-2200; debug/chat_demo_with_kvcache.tl:44-88.)
// O is multiplied by e^(old maximum - new maximum) only where some row of a warp has a new maximum; elsewhere the
// factor is exactly one.
//
// Warps:  0  Q, K and V by TMA      1  tensor memory and MMA issue      2-5  softmax, rescale, output
//
// Keys past the last query of the sequence lie outside the tensor maps and read as zero.
// What it measured, against the mma.sync kernel of 64 rows per CTA it replaces: 2048 tokens, 32 heads of 128 (7B)
// 250 -> 64 us (536 TFLOP/s of the visible half of the scores); 32 heads over 4 KV heads of 64 (TinyLlama) 130 -> 54 us,
// 512 tokens 21.8 -> 14.2; 32 tokens after 1000 27.7 -> 20.3; 64 tokens and fewer 3 to 5 us as before.  The results
// are the same to the last bit (the same products in the same order, the same maxima and exponentials).  It is bound by
// the softmax: about 13 instructions a score, half of them expf.  (Two cheaper forms measured 40 us at the first size
// and are not used: an exponential from one fused multiply-add and ex2, and a maximum followed only when it has risen
// by e^5, which rounds P differently.  Two threads a row, with half the registers each: 76 us.)
//
// All waits are bounded; one that runs out sets the status word and lets the CTA drain, free its tensor
// memory and return.
#include <cuda.h>

#include "tlc_attention_tc.h"
#include "tlc_gemm_kernel.cuh"

using namespace tlc_gemm;

namespace {

constexpr int kRows = 128, kKeys = 64, kThreads = 192;
constexpr int kHalf = kKeys * 128;  // bytes of 64 keys x 64 values
template <int D> constexpr int kv_bytes() { return kHalf * (D / 64); }
// K and V tiles in flight: what two CTAs an SM leave room for
template <int D> constexpr int stages() { return D == 128 ? 2 : 3; }
template <int D> constexpr int smem_bytes_tc() { return 1024 + 1024 + kRows * D * 2 + 2 * stages<D>() * kv_bytes<D>(); }
constexpr int kTmemCols = 256;  // scores: two tiles of 64 columns; O: D
constexpr int kColO = 128;

struct FlashParams {
    __half *out;
    int I, H, Hkv, G;
    int q_tiles, batch;
    int splits;  // CTAs (of one cluster) that share a tile's keys
    int pos0;
    float scale;
    tlc_dev_status *status;
    uint64_t wait_ns;
};

__device__ __forceinline__ void tma_load_3d_el(uint32_t dst, const void *map, int x, int y, int z, uint32_t bar, uint32_t el) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %6, 0;\n"
        " @q cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n}\n" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar), "r"(el)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d_el(uint32_t dst, const void *map, int x, int y, int z, int w, uint32_t bar, uint32_t el) {
    asm volatile(
        "{\n .reg .pred q;\n setp.ne.b32 q, %7, 0;\n"
        " @q cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n}\n" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar), "r"(el)
        : "memory");
}
// Columns of this thread's lane.  The load is waited for by tmem_ld_wait, which the registers pass through: nothing
// that uses them can be moved in front of it.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&a)[32], uint32_t (&b)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int e = 0; e < 32; e++) asm volatile("" : "+r"(a[e]), "+r"(b[e]));
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

static_assert(kRows * (64 + 2) * 4 <= kRows * 64 * 2 + 2 * stages<64>() * kv_bytes<64>() &&
                  kRows * (128 + 2) * 4 <= kRows * 128 * 2 + 2 * stages<128>() * kv_bytes<128>(),
              "the merge takes the place of Q, K and V");
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t at, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}

template <int D>
__global__ void __launch_bounds__(kThreads, 2)
    attention_tc_kernel(const __grid_constant__ FlashParams p, const __grid_constant__ CUtensorMap q_map,
                        const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map) {
    constexpr int HALVES = D / 64, ST = stages<D>(), KV = kv_bytes<D>();
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t *k_full = reinterpret_cast<uint64_t *>(base), *k_empty = k_full + ST, *v_full = k_empty + ST, *v_empty = v_full + ST;
    uint64_t *s_full = v_empty + ST, *p_full = s_full + 2, *pv_done = p_full + 2, *q_full = pv_done + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(q_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    uint8_t *qs = base + 1024, *ks = qs + kRows * D * 2, *vs = ks + ST * KV;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < ST; i++) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4);
            mbar_init(&pv_done[i], 1);
        }
        mbar_init(q_full, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // The last queries of a sequence see the most keys: their tiles go first.
    const int split = blockIdx.x % p.splits, cta = blockIdx.x / p.splits;
    const int per = p.Hkv * p.batch, hb = cta % per, qt = p.q_tiles - 1 - cta / per;
    const int hk = hb % p.Hkv, b = hb / p.Hkv;
    const int G = p.G, RQ = kRows / G;
    const int k_end = p.pos0 + min(p.I, (qt + 1) * RQ);
    // key tiles of this CTA: [t0, t0 + n)
    const int tiles = (k_end + kKeys - 1) / kKeys, share = (tiles + p.splits - 1) / p.splits, t0 = split * share;
    const int n = max(0, min(tiles - t0, share));

    if (warp == 0) {
        // ------------------------------ Q, K, V ------------------------------
        // (Dependents are let in when this CTA has its tensor memory: theirs must not be asked for first.)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint32_t el = elect_one();
        const uint32_t bar_q = smem_u32(q_full);
        if (n > 0) mbar_arrive_expect_tx_el(q_full, kRows * D * 2, el);
#pragma unroll
        for (int h = 0; h < HALVES; h++)
            if (n > 0) tma_load_3d_el(smem_u32(qs + h * kRows * 128), &q_map, 64 * h, hk * G, b * p.I + qt * RQ, bar_q, el);
        bool ok = true;
        int sk = 0, sv = 0;
        uint32_t pk = 1, pv = 1;
        for (int j = 0; ok && n > 0 && j <= n; j++) {  // K of tile j, V of tile j - 1: the order in which they are used
            if (j < n) {
                ok = __all_sync(0xffffffffu, mbar_wait(&k_empty[sk], pk, abort_flag, p.status, 41, p.wait_ns));
                if (!ok) break;
                const uint32_t bar = smem_u32(&k_full[sk]);
                mbar_arrive_expect_tx_el(&k_full[sk], KV, el);
#pragma unroll
                for (int h = 0; h < HALVES; h++)
                    tma_load_4d_el(smem_u32(ks + sk * KV + h * kHalf), &k_map, 64 * h, hk, (t0 + j) * kKeys, b, bar, el);
                if (++sk == ST) sk = 0, pk ^= 1u;
            }
            if (j > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait(&v_empty[sv], pv, abort_flag, p.status, 42, p.wait_ns));
                if (!ok) break;
                const uint32_t bar = smem_u32(&v_full[sv]);
                mbar_arrive_expect_tx_el(&v_full[sv], KV, el);
#pragma unroll
                for (int h = 0; h < HALVES; h++)
                    tma_load_4d_el(smem_u32(vs + sv * KV + h * kHalf), &v_map, 64 * h, hk, (t0 + j - 1) * kKeys, b, bar, el);
                if (++sv == ST) sv = 0, pv ^= 1u;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------ MMA ------------------------------
        const uint32_t el = elect_one();
        const uint32_t idesc_s = idesc_for(kKeys), idesc_o = idesc_for(D) | 1u << 16;  // (V: N-major)
        constexpr uint32_t MN = (uint32_t)(kHalf >> 4) << 16;  // the next 64 values of d: the next box
        const uint32_t q0 = (smem_u32(qs) & 0x3FFFF) >> 4, k0 = (smem_u32(ks) & 0x3FFFF) >> 4, v0 = (smem_u32(vs) & 0x3FFFF) >> 4;
        bool ok = n > 0 && mbar_wait(q_full, 0, abort_flag, p.status, 43, p.wait_ns);
        int sk = 0, sv = 0;
        uint32_t pk = 0, pv = 0;
        auto scores = [&](int j) {  // S of tile j
            ok = mbar_wait(&k_full[sk], pk, abort_flag, p.status, 44, p.wait_ns) && ok;
            // its columns hold P of tile j - 2
            if (j >= 2) ok = mbar_wait(&pv_done[j & 1], (uint32_t)((j - 2) >> 1) & 1u, abort_flag, p.status, 45, p.wait_ns) && ok;
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            if (ok) {
                const uint32_t at = tmem + (j & 1) * kKeys, kd = k0 + sk * (KV >> 4);
#pragma unroll
                for (int k16 = 0; k16 < D / 16; k16++)
                    umma_f16(at, desc_at(q0 + (k16 >> 2) * (kRows * 128 >> 4) + (k16 & 3) * 2),
                             desc_at(kd + (k16 >> 2) * (kHalf >> 4) + (k16 & 3) * 2), idesc_s, k16 > 0, el);
            }
            umma_commit(&k_empty[sk], el);
            umma_commit(&s_full[j & 1], el);
            if (++sk == ST) sk = 0, pk ^= 1u;
        };
        if (n > 0) scores(0);
        for (int j = 0; j < n; j++) {
            if (j + 1 < n) scores(j + 1);
            ok = mbar_wait(&v_full[sv], pv, abort_flag, p.status, 46, p.wait_ns) && ok;
            ok = mbar_wait(&p_full[j & 1], (uint32_t)(j >> 1) & 1u, abort_flag, p.status, 47, p.wait_ns) && ok;
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            if (ok) {
                const uint32_t at = tmem + (j & 1) * kKeys, vd = v0 + sv * (KV >> 4);
#pragma unroll
                for (int k16 = 0; k16 < kKeys / 16; k16++)
                    umma_f16_ts(tmem + kColO, at + k16 * 8, (desc_at(vd + k16 * 128) & ~(uint64_t)(1u << 16)) | MN, idesc_o,
                                (j > 0 || k16 > 0) ? 1u : 0u, el);
            }
            umma_commit(&v_empty[sv], el);
            umma_commit(&pv_done[j & 1], el);
            if (++sv == ST) sv = 0, pv ^= 1u;
        }
        __syncwarp();
    } else {
        // ------------------------------ softmax ------------------------------
        const int quarter = warp & 3, r = 32 * quarter + lane;
        const uint32_t tl = tmem + ((uint32_t)(32 * quarter) << 16);
        const int qi = qt * RQ + r / G, head = hk * G + r % G;
        const int last = min(p.pos0 + qi, k_end - 1);  // last key this row sees; below, what the warp's rows see
        const int warp_first = p.pos0 + qt * RQ + 32 * quarter / G;
        const int warp_last = warp_first < p.pos0 + p.I ? min(p.pos0 + qt * RQ + (32 * quarter + 31) / G, k_end - 1) : -1;
        const __half2 scale2 = __float2half2_rn(p.scale);
        const __half neg_inf = __float2half_rn(-INFINITY);
        // The row's sum in four parts (pairs of keys in turn), each in the order of the keys.
        float m_run = -INFINITY, l_run[4] = {0.f, 0.f, 0.f, 0.f};
        for (int j = 0; j < n; j++) {
            const int j0 = (t0 + j) * kKeys;
            const uint32_t ts = tl + (j & 1) * kKeys;
            mbar_wait(&s_full[j & 1], (uint32_t)(j >> 1) & 1u, abort_flag, p.status, 48, p.wait_ns);
            __syncwarp();
            tc_fence_after();
            uint32_t pk[32];
            const int seen = warp_last - j0;  // (warp-uniform) keys past it count for no row of the warp
            if (seen < 0) {
#pragma unroll
                for (int e = 0; e < 32; e++) pk[e] = 0u;
            } else {
                __half2 v[32];
                {
                    uint32_t s0[32], s1[32];
                    tmem_ld32_issue(ts, s0);
                    tmem_ld32_issue(ts + 32, s1);
                    tmem_ld_wait(s0, s1);
#pragma unroll
                    for (int e = 0; e < 16; e++) {
                        v[e] = __hmul2(__floats2half2_rn(__uint_as_float(s0[2 * e]), __uint_as_float(s0[2 * e + 1])), scale2);
                        v[16 + e] = __hmul2(__floats2half2_rn(__uint_as_float(s1[2 * e]), __uint_as_float(s1[2 * e + 1])), scale2);
                    }
                }
                if (j0 + kKeys > k_end || j0 + kKeys - 1 > warp_first) {
#pragma unroll
                    for (int e = 0; e < 32; e++) {
                        if (2 * e > last - j0) v[e].x = neg_inf;
                        if (2 * e + 1 > last - j0) v[e].y = neg_inf;
                    }
                }
                __half2 m4[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
                for (int e = 4; e < 32; e++) m4[e & 3] = __hmax2(m4[e & 3], v[e]);
                const __half2 mh = __hmax2(__hmax2(m4[0], m4[1]), __hmax2(m4[2], m4[3]));
                const float m_new = fmaxf(m_run, fmaxf(__low2float(mh), __high2float(mh)));
                const float m_safe = m_new == -INFINITY ? 0.f : m_new;
                const bool moved = m_new > m_run;
                const float corr = expf(m_run - m_safe);
                m_run = m_new;
                float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (16 * c > seen) {
#pragma unroll
                        for (int e = 8 * c; e < 8 * c + 8; e++) pk[e] = 0u;
                        continue;
                    }
#pragma unroll
                    for (int e = 8 * c; e < 8 * c + 8; e++) {
                        const float2 f = __half22float2(v[e]);
                        const float a = expf(f.x - m_safe), d = expf(f.y - m_safe);
                        sum[e & 3] += a;
                        sum[e & 3] += d;
                        const __half2 h = __floats2half2_rn(a, d);
                        pk[e] = *reinterpret_cast<const uint32_t *>(&h);
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; e++) l_run[e] = l_run[e] * corr + sum[e];
                if (j > 0 && __any_sync(0xffffffffu, moved)) {
                    mbar_wait(&pv_done[(j - 1) & 1], (uint32_t)((j - 1) >> 1) & 1u, abort_flag, p.status, 49, p.wait_ns);
                    __syncwarp();
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < D; c += 64) {
                        uint32_t o[32], o2[32];
                        tmem_ld32_issue(tl + kColO + c, o);
                        tmem_ld32_issue(tl + kColO + c + 32, o2);
                        tmem_ld_wait(o, o2);
#pragma unroll
                        for (int e = 0; e < 32; e++) {
                            o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
                            o2[e] = __float_as_uint(__uint_as_float(o2[e]) * corr);
                        }
                        tmem_st32(tl + kColO + c, o);
                        tmem_st32(tl + kColO + c + 32, o2);
                    }
                }
            }
            tmem_st32(ts, pk);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[j & 1]);
        }
        const bool ok = n == 0 || mbar_wait(&pv_done[(n - 1) & 1], (uint32_t)((n - 1) >> 1) & 1u, abort_flag, p.status, 50, p.wait_ns);
        __syncwarp();
        tc_fence_after();
        const float l = (l_run[0] + l_run[1]) + (l_run[2] + l_run[3]);
        if (p.splits == 1) {
            const float inv = l > 0.f ? 1.0f / l : 0.f;
            __half *out = p.out + ((size_t)(b * (size_t)p.I + qi) * p.H + head) * D;
#pragma unroll
            for (int c = 0; c < D; c += 64) {
                uint32_t o[2][32];
                tmem_ld32_issue(tl + kColO + c, o[0]);
                tmem_ld32_issue(tl + kColO + c + 32, o[1]);
                tmem_ld_wait(o[0], o[1]);
                if (ok && qi < p.I) {
#pragma unroll
                    for (int e = 0; e < 64; e += 8) {
                        __align__(16) __half2 h[4];
#pragma unroll
                        for (int i = 0; i < 8; i += 2)
                            h[i / 2] = __floats2half2_rn(__uint_as_float(o[e / 32][e % 32 + i]) * inv,
                                                         __uint_as_float(o[e / 32][e % 32 + i + 1]) * inv);
                        *reinterpret_cast<uint4 *>(out + c + e) = *reinterpret_cast<const uint4 *>(h);
                    }
                }
                __syncwarp();
            }
        } else {
            // The CTAs of the cluster are done with their tiles, whose place now takes what the owner of a row
            // adds up: [split][O, maximum, sum][row], so that the rows of a warp lie side by side.
            cluster_barrier();
            const int own = kRows / p.splits, owner = r / own, pitch = (D + 2) * own;
            uint32_t to;
            asm("mapa.shared::cluster.u32 %0, %1, %2;"
                : "=r"(to)
                : "r"(smem_u32(qs) + (uint32_t)(split * pitch + r - owner * own) * 4), "r"(owner));
            st_cluster(to + D * own * 4, n == 0 ? 0xFF800000u : __float_as_uint(m_run));  // (-inf: no keys here)
            st_cluster(to + (D + 1) * own * 4, __float_as_uint(l));
            if (n > 0)
#pragma unroll
                for (int c = 0; c < D; c += 32) {
                    uint32_t o[32];
                    tmem_ld32(tl + kColO + c, o);
#pragma unroll
                    for (int e = 0; e < 32; e++) st_cluster(to + (c + e) * own * 4, o[e]);
                    __syncwarp();
                }
            cluster_barrier();
            // `splits` threads a row, D / splits values each (8 at least)
            const int row = r % own, mine = split * own + row, d0 = r / own * (D / p.splits);
            const float *part = reinterpret_cast<const float *>(qs) + row;
            const int oq = qt * RQ + mine / G;
            float M = -INFINITY, L = 0.f, w[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (i < p.splits) M = fmaxf(M, part[i * pitch + D * own]);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                w[i] = 0.f;
                if (i < p.splits) {
                    const float mi = part[i * pitch + D * own];
                    if (mi > -INFINITY) w[i] = expf(mi - M);
                    L += part[i * pitch + (D + 1) * own] * w[i];
                }
            }
            const float inv = L > 0.f ? 1.0f / L : 0.f;
            __half *out = p.out + ((size_t)(b * (size_t)p.I + oq) * p.H + hk * G + mine % G) * D + d0;
            for (int d = 0; d < D / p.splits; d += 8) {
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (i < p.splits && w[i] > 0.f)  // (a split without keys has stored no O)
#pragma unroll
                        for (int e = 0; e < 8; e++) acc[e] += part[i * pitch + (d0 + d + e) * own] * w[i];
                if (ok && oq < p.I) {
                    __align__(16) __half2 h[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) h[e] = __floats2half2_rn(acc[2 * e] * inv, acc[2 * e + 1] * inv);
                    *reinterpret_cast<uint4 *>(out + d) = *reinterpret_cast<const uint4 *>(h);
                }
            }
        }
        __syncwarp();
        tc_fence_before();
    }
    if (p.splits > 1 && warp < 2) {  // (every thread of the cluster takes part in its two barriers)
        __syncwarp();
        cluster_barrier();
        cluster_barrier();
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmemCols) : "memory");
    }
}

template <int D>
int32_t launch(tlc_ctx *ctx, const FlashParams &p, const CUtensorMap &q, const CUtensorMap &k, const CUtensorMap &v) {
    static bool configured[64] = {};
    if (!configured[ctx->device & 63]) {
        TLC_CUDA(cudaFuncSetAttribute(attention_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes_tc<D>()));
        TLC_CUDA(cudaFuncSetAttribute(attention_tc_kernel<D>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      cudaSharedmemCarveoutMaxShared));
        configured[ctx->device & 63] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.q_tiles * p.Hkv * p.batch * p.splits));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_bytes_tc<D>();
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (p.splits > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)p.splits;
        attr[na].val.clusterDim.y = 1;
        attr[na++].val.clusterDim.z = 1;
    }
    if (ctx->use_pdl && ctx->pdl_small) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t le = cudaLaunchKernelEx(&cfg, attention_tc_kernel<D>, p, q, k, v);
    if (le != cudaSuccess) {
        cudaGetLastError();
        return tlc_fail(TLC_ERR_CUDA, "attention launch failed: %s", cudaGetErrorString(le));
    }
    TLC_CHECK_LAUNCH(ctx);
    return TLC_OK;
}

}  // namespace

bool tlc_attention_tc_maps(AttnTc &a) {
    if (((uintptr_t)a.out & 15) != 0) return false;
    const uint64_t D = a.D, row = (uint64_t)a.H * D * 2, kv = (uint64_t)a.Hkv * D * 2;
    const uint64_t qd[3] = {D, (uint64_t)a.H, (uint64_t)a.batch * a.I}, qst[2] = {D * 2, row};
    const uint32_t qb[3] = {64, (uint32_t)(a.H / a.Hkv), (uint32_t)(kRows / (a.H / a.Hkv))};
    const uint64_t kd[4] = {D, (uint64_t)a.Hkv, (uint64_t)(a.pos0 + a.I), (uint64_t)a.batch}, kst[3] = {D * 2, kv, kv * a.Tmax};
    const uint32_t kb[4] = {64, 1, kKeys, 1};
    return encode_map_nd(&a.q_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, a.q, 3, qd, qst, qb) &&
           encode_map_nd(&a.k_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, a.kc, 4, kd, kst, kb) &&
           encode_map_nd(&a.v_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, a.vc, 4, kd, kst, kb);
}

int32_t tlc_launch_attention_tc(tlc_ctx *ctx, const AttnTc &a) {
    FlashParams p{};
    p.out = a.out;
    p.I = a.I;
    p.H = a.H;
    p.Hkv = a.Hkv;
    p.G = a.H / a.Hkv;
    p.q_tiles = (a.I + kRows / p.G - 1) / (kRows / p.G);
    p.batch = a.batch;
    p.pos0 = a.pos0;
    // A short prompt behind a long context has few tiles of rows, each with many keys: the keys are shared out over
    // the CTAs of a cluster, up to two CTAs an SM, by the microseconds of a CTA's key tiles, of the merge (3 to 5) and
    // of what the next kernel's CTAs lose, which would have fetched weights on the idle SMs (4).  32 heads over 4 KV
    // heads of 64: 32 tokens after 1000 20.7 us, 8 splits 10.1; 300 after 1000 28.2, 2 splits 22.6; 32 heads of 128, 128
    // tokens after 1900 42.0, now 18.5.  TinyLlama, 20 tokens after 1500: 1.65 -> 1.35 ms; 77 after 391, where the kernel
    // alone gains 2 us from 8 splits, the same.
    const int ctas = p.q_tiles * p.Hkv * p.batch, tiles = (a.pos0 + a.I + kKeys - 1) / kKeys;
    p.splits = 1;
    double best = tiles * 0.95;
    for (int s = 2; s <= 8 && ctas * s <= 2 * ctx->sm_count; s *= 2) {
        const double t = (tiles + s - 1) / s * (ctas * s > ctx->sm_count ? 1.2 : 0.95) + (a.D == 64 ? 7.2 : 8.7);
        if (t < best) {
            best = t;
            p.splits = s;
        }
    }
    p.scale = a.scale;
    p.status = ctx->dev_status;
    p.wait_ns = ctx->wait_ns;
    return a.D == 64 ? launch<64>(ctx, p, a.q_map, a.k_map, a.v_map) : launch<128>(ctx, p, a.q_map, a.k_map, a.v_map);
}
