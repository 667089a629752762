// The fused dequant-GEMV kernel for 2 to 16 activation rows.  See tlc_gemv.cu for the design notes.
#pragma once

#include "tlc_gemv_common.cuh"

namespace tlc_gemv {

// What a consumer warp holds the activations of, in registers, for the whole launch: TI = 1, 2, 3 times 128 columns
// (Q4_0: TI tiles, Q8_0: 2 TI tiles); Q6_K: one super-block of 256 columns (TI = 1).
template <int QT> constexpr int tiles_of(int ti) { return QT == TLC_TYPE_Q6_K ? 1 : ti * (QT == TLC_TYPE_Q4_0 ? 1 : 2); }
// Accumulator start values of a warp's window: one per 32 columns, Q6_K one per 16.
template <int QT> constexpr int starts_of(int ti) { return QT == TLC_TYPE_Q6_K ? 16 : 4 * ti; }
// Q6_K: a slab is fetched in boxes of eight super-blocks; a row of a box takes 16 bytes of the next super-block
// along, so that the rows of a fragment lie in different banks.
constexpr int kQ6BoxRow = 8 * 224 + 16, kQ6Box = 16 * kQ6BoxRow;

constexpr int kRedPitch = 20;  // f32 per activation row of a warp's 16 sums: the lanes' stores meet 32 banks

// Shared-memory layout (bytes from the start of dynamic shared memory):
//   0     full [8], empty [8] mbarriers          128 abort flag
//   256   cinit: accumulator start values [CW warps][4 TI blocks, or 16 groups][8 NT] f32
//   ...   red   [2][batch][CW warps][8 NT rows][20] f32
//   ...   part  [round][8 NT][16] f32: a cluster CTA's share of the sums
//   ...   ring  [stages][tiles of the CTA's window] weight tiles as they lie in HBM (128-byte aligned)
struct GemvSmem {
    int red, part, ring, red_slot;
};
__host__ __device__ inline GemvSmem gemv_smem(int cw, int starts, int nt, int batch, int round) {
    GemvSmem s;
    s.red = 256 + cw * starts * 8 * nt * 4;
    s.red_slot = cw * 8 * nt * kRedPitch;
    s.part = s.red + 2 * batch * s.red_slot * 4;
    s.ring = (s.part + round * 8 * nt * 16 * 4 + 127) & ~127;
    return s;
}

// Activations in fragment order, as frag_rows_kernel leaves them: [block][row tile of 8][lane] 16 bytes, lane
// (g, t) holding eight values of row g; behind them the start values [block][8 row tiles' rows] f32.
__host__ __device__ inline size_t frag_bytes(int64_t nblk, int nt) { return (size_t)nblk * nt * 512; }
__host__ __device__ inline size_t frag_total_bytes(int64_t nblk, int nt) { return frag_bytes(nblk, nt) + (size_t)nblk * nt * 32; }
// Eight values of lane t of a block, as they lie in the row -> fragment order.
//   Q4_0: {4t .. 4t+3, 16+4t .. 19+4t} -> {4t, 4t+2, 16+4t, 18+4t | 4t+1, 4t+3, 17+4t, 19+4t}
//   Q8_0: {8t .. 8t+7}, as they lie
template <int QT>
__device__ __forceinline__ uint4 load_piece(const __half *blk, int t) {
    if (QT == TLC_TYPE_Q4_0) {
        const uint2 lo = *reinterpret_cast<const uint2 *>(blk + 4 * t), hi = *reinterpret_cast<const uint2 *>(blk + 16 + 4 * t);
        return make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
    return *reinterpret_cast<const uint4 *>(blk + 8 * t);
}
template <int QT>
__device__ __forceinline__ uint4 to_fragment(const uint4 &v) {
    if (QT != TLC_TYPE_Q4_0) return v;
    return make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410), __byte_perm(v.x, v.y, 0x7632),
                      __byte_perm(v.z, v.w, 0x7632));
}
// -OFFSET * sum of a block's activations * 2^-24 from a piece in fragment order (all lanes of the quad get it).
template <int QT>
__device__ __forceinline__ float start_value(const uint4 &f) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&f.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&f.y));
    const float2 c = __half22float2(*reinterpret_cast<const __half2 *>(&f.z)), d = __half22float2(*reinterpret_cast<const __half2 *>(&f.w));
    float s = ((a.x + a.y) + (b.x + b.y)) + ((c.x + c.y) + (d.x + d.y));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return -QTraits<QT>::OFFSET * 5.9604644775390625e-08f * s;
}

// RMSNorm of the activation rows and their fragment order, once per call instead of once per CTA of the GEMV
// (8 rows of K = 8192: the GEMV's CTAs took 8 us over it, more than over the weights of a TP8 rank's
// projection).  One CTA per row; rows past m are written as zeros.  Bound by the latency of one pass over the row.
// W_EARLY: see norm_early of tlc_gemv_args.
template <int QT, bool W_EARLY>
__global__ void __launch_bounds__(512) frag_rows_kernel(const __half *x, const __half *w, int m, int k,
                                                        float eps, uint4 *__restrict__ frag, float *__restrict__ start, int nt) {
    __shared__ float part[16];
    constexpr int KEEP = 4;  // pieces of the row a thread keeps: K = 16384
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, items = k / 8;
    const __half *xr = x + (size_t)row * k;
    uint4 nw = make_uint4(0, 0, 0, 0);
    if (W_EARLY && tid < items) nw = load_piece<QT>(w + (tid >> 2) * 32, tid & 3);
    tlc_pdl_after_wait();
    if (!W_EARLY && tid < items) nw = load_piece<QT>(w + (tid >> 2) * 32, tid & 3);
    const bool live = row < m;
    uint4 v[KEEP];
    float sq = 0.f;
    auto add = [&](const uint4 &u) {
        const __half2 *h = reinterpret_cast<const __half2 *>(&u);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(h[j]);
            sq = fmaf(f.x, f.x, sq);
            sq = fmaf(f.y, f.y, sq);
        }
    };
#pragma unroll
    for (int r = 0; r < KEEP; r++) {
        const int i = tid + r * 512;
        v[r] = live && i < items ? load_piece<QT>(xr + (i >> 2) * 32, i & 3) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int r = 0; r < KEEP; r++) add(v[r]);
    for (int i = tid + KEEP * 512; i < items; i += 512)
        if (live) add(load_piece<QT>(xr + (i >> 2) * 32, i & 3));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if (lane == 0) part[tid >> 5] = sq;
    __syncthreads();
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 16; i++) ss += part[i];
    const float inv = 1.0f / sqrtf(ss / (float)k + eps);
    auto emit = [&](int i, const uint4 &raw, const uint4 &wv) {
        // f16((x * inv) * w): two separately rounded f32 multiplies, then RNE
        // (Tensor::rms_norm_cpu, src/ops/normalization.rs:236-240)
        const __half2 *xh = reinterpret_cast<const __half2 *>(&raw), *wh = reinterpret_cast<const __half2 *>(&wv);
        __half2 o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(xh[j]), g = __half22float2(wh[j]);
            o[j] = __floats2half2_rn(__fmul_rn(__fmul_rn(f.x, inv), g.x), __fmul_rn(__fmul_rn(f.y, inv), g.y));
        }
        const uint4 f = to_fragment<QT>(*reinterpret_cast<const uint4 *>(o));
        const float cv = start_value<QT>(f);
        const int b = i >> 2, t = i & 3;
        if (i < items) {
            frag[((size_t)b * nt + (row >> 3)) * 32 + (row & 7) * 4 + t] = f;
            if (t == 0) start[(size_t)b * nt * 8 + row] = cv;
        }
    };
    for (int r = 0; r * 512 < items; r++) {
        const int i = tid + r * 512;
        const bool in = live && i < items;
        uint4 raw = make_uint4(0, 0, 0, 0), wv = nw;
        if (r < KEEP) {
#pragma unroll
            for (int q = 0; q < KEEP; q++)
                if (q == r) raw = v[q];
        } else if (in) {
            raw = load_piece<QT>(xr + (i >> 2) * 32, i & 3);
        }
        if (r > 0) wv = in ? load_piece<QT>(w + (i >> 2) * 32, i & 3) : make_uint4(0, 0, 0, 0);
        emit(i, raw, wv);
    }
}

// Bounded wait of a whole warp.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, tlc_dev_status *status,
                                          int where, uint64_t wait_ns) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, where, wait_ns));
}

// NT: column tiles of eight activation rows.  TI: see tiles_of.  CW: consumer warps, 8 (two CTAs per
// SM) or 16 (one).  The activations come as rows (p.x) or in fragment order (p.frag, normalised).
template <int QT, int NT, int TI, int CW>
__global__ void __launch_bounds__(CW * 32, CW == 8 ? 2 : 1) gemv_mma_kernel(const __grid_constant__ GemvParams p) {
    using T = QTraits<QT>;
    constexpr int CT = CW * 32;
    constexpr int TILE = T::TILE_BYTES;
    constexpr int TW = tiles_of<QT>(TI);  // tiles of a warp's window
    constexpr bool Q6 = QT == TLC_TYPE_Q6_K;
    constexpr int NB = starts_of<QT>(TI);  // blocks (Q6_K: groups of 16)
    constexpr int BK = Q6 ? 16 : 32;       // columns of a block
    constexpr int NR = Q6 ? 2 : 4;         // fragment registers of a block
    constexpr int MP = 8 * NT;

    extern __shared__ __align__(128) uint8_t smem[];
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 128);
    const GemvSmem lay = gemv_smem(CW, NB, NT, p.batch, p.round);
    float *cinit = reinterpret_cast<float *>(smem + 256);
    float *red = reinterpret_cast<float *>(smem + lay.red);
    float *part = reinterpret_cast<float *>(smem + lay.part);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int S = p.nstages;
    // The K range is shared out over the ks CTAs of a cluster and, inside a CTA, over the warps.
    const int ks = p.ksplit;
    const int rank = ks > 1 ? (int)blockIdx.x % ks : 0, cta_i = ks > 1 ? (int)blockIdx.x / ks : (int)blockIdx.x;
    const int cta_n = ks > 1 ? (int)gridDim.x / ks : (int)gridDim.x;
    const int kt0 = rank * p.ktiles_win;                                    // first tile of the CTA's window
    const int my_ktiles = max(0, min(p.ktiles_win, p.ktiles - kt0));

    // Units of this CTA, worked out before anything waits for the previous kernel.
    const int u_lo = p.contig ? (int)((long long)cta_i * p.total_units / cta_n) : 0;
    const int u_hi = p.contig ? (int)((long long)(cta_i + 1) * p.total_units / cta_n) : 0;
    const int n_mine = p.contig ? u_hi - u_lo : ((int)p.total_units - cta_i + cta_n - 1) / cta_n;
    auto unit_at = [&](int i) { return p.contig ? u_lo + i : cta_i + i * cta_n; };
    // unit (of one slab) -> weight and slab
    auto place = [&](int unit, int &ti, int &sl) {
        ti = 0;
        sl = unit;
        if (p.subs == 1) {
            if (sl >= p.slabs[0]) { sl -= p.slabs[0]; ti = 1; }
            if (ti == 1 && sl >= p.slabs[1]) { sl -= p.slabs[1]; ti = 2; }
        }
    };

    const int g = lane >> 2, t = lane & 3;
    const int kb0 = kt0 * T::TB;                                                        // first block of the CTA's window
    const int wt0 = warp * p.tiles_warp;                                                // first tile of the warp, in the window
    const int my_tiles = max(0, min(p.tiles_warp, my_ktiles - wt0));
    const int wb0 = kb0 + wt0 * T::TB;                                                  // first block of the warp
    const int my_blocks = max(0, min(my_tiles * T::TB, p.k / BK - wb0));                // blocks that exist

    // A ring of slabs (the CTA's window of each: one bulk copy, its tiles lie side by side).  There is no
    // producer warp -- its registers are worth more in the consumers -- : the warps take turns, one slab
    // each, in refilling the stage of the slab before.  One copy per slab and not one per warp: a
    // bulk copy takes its SM about 150 clocks whatever its size.  Weights are never written by a
    // kernel, so the ring fills before the previous kernel of the stream has finished.
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + 8;
    const uint32_t ring = smem_u32(smem + lay.ring);
    const uint32_t copy_bytes = (uint32_t)(my_ktiles * TILE);
    const int n_slabs = my_ktiles > 0 ? n_mine * p.subs : 0;
    auto fetch = [&](int i, int s) {  // slab i of this CTA into stage s (one lane)
        if (i >= n_slabs) return;
        int ti, sl;
        place(unit_at(p.subs == 2 ? i >> 1 : i), ti, sl);
        const int tw = p.subs == 2 ? i & 1 : ti;
        if constexpr (Q6) {
            const int boxes = (my_ktiles + 7) >> 3;
            mbar_expect_tx(&full[s], (uint32_t)(boxes * kQ6Box));
            for (int b = 0; b < boxes; b++)  // (the map counts in 8-byte elements)
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                        ring + (uint32_t)(s * p.stage_bytes + b * kQ6Box)),
                    "l"(reinterpret_cast<uint64_t>(p.w_map)), "r"((kt0 + 8 * b) * 28), "r"(sl * kRows), "r"(smem_u32(&full[s]))
                    : "memory");
            return;
        }
        const uint8_t *src = p.t[tw].w + (size_t)sl * p.t[tw].slab_pitch + (size_t)kt0 * TILE;
        mbar_expect_tx(&full[s], copy_bytes);
        bulk_g2s_hint(smem + lay.ring + (size_t)s * p.stage_bytes, src, copy_bytes, &full[s], l2_evict_first_policy());
    };
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CW);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (ks > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // (waited for before the first remote access)
    __syncthreads();
    if (p.pdl_mode == 1) pdl_launch_dependents();
    if (warp == CW - 1 && lane == 0)
        for (int s = 0; s < S; s++) fetch(s, s);
    __syncwarp();
    pdl_wait();  // the activations (and residual) come from the previous kernel
    if (p.pdl_mode == 3) pdl_launch_dependents();

    // (a) The warp's window of the activations into fragment registers (lane (g, t): eight values of every block
    // of row g (+ 8)), and the accumulator start values to shared memory.
    uint32_t xb[NT][NB][NR];
    float *ci_w = cinit + warp * NB * MP;
    if constexpr (Q6) {
        // lane (g, t): elements 4t .. 4t+3 of every group of 16 of row g, as they lie
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const int m = nt * 8 + g;
            const __half *xr = p.x + (size_t)(m < p.m ? m : 0) * p.k + (size_t)wb0 * 16 + 4 * t;
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const uint2 v = b < my_blocks && m < p.m ? *reinterpret_cast<const uint2 *>(xr + b * 16) : make_uint2(0, 0);
                xb[nt][b][0] = v.x;
                xb[nt][b][1] = v.y;
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&xb[nt][b][0]));
                const float2 c = __half22float2(*reinterpret_cast<const __half2 *>(&xb[nt][b][1]));
                float s = (a.x + a.y) + (c.x + c.y);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                if (t == 0) ci_w[b * MP + nt * 8 + g] = -32.0f * 5.9604644775390625e-08f * s;  // * 2^-24
            }
    } else if (p.frag) {
#pragma unroll
        for (int b = 0; b < NB; b++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const uint4 v = b < my_blocks ? p.frag[((size_t)(wb0 + b) * NT + nt) * 32 + lane] : make_uint4(0, 0, 0, 0);
                xb[nt][b][0] = v.x;
                xb[nt][b][1] = v.y;
                xb[nt][b][2] = v.z;
                xb[nt][b][3] = v.w;
            }
        for (int i = lane; i < NB * MP; i += 32) ci_w[i] = i < my_blocks * MP ? p.start[(size_t)wb0 * MP + i] : 0.f;
    } else {
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const int m = nt * 8 + g;
            const __half *xr = p.x + (size_t)(m < p.m ? m : 0) * p.k + (size_t)wb0 * 32;
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const uint4 v = b < my_blocks && m < p.m ? load_piece<QT>(xr + b * 32, t) : make_uint4(0, 0, 0, 0);
                xb[nt][b][0] = v.x;
                xb[nt][b][1] = v.y;
                xb[nt][b][2] = v.z;
                xb[nt][b][3] = v.w;
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const uint4 f = to_fragment<QT>(make_uint4(xb[nt][b][0], xb[nt][b][1], xb[nt][b][2], xb[nt][b][3]));
                const float cv = start_value<QT>(f);
                if (t == 0) ci_w[b * MP + nt * 8 + g] = cv;
                xb[nt][b][0] = f.x;
                xb[nt][b][1] = f.y;
                xb[nt][b][2] = f.z;
                xb[nt][b][3] = f.w;
            }
    }
    __syncwarp();
    const uint32_t ci_addr = smem_u32(ci_w + 2 * t);

    // Outputs are handed out as (pair q of unit and activation row, row of the slab): row = tid & 15, q = tid >> 4
    // and up; q / m by a multiplication (q < 4096).
    const int row16 = tid & 15;
    auto split_q = [&](int q, int &ui, int &col) {
        ui = (q * p.m_inv) >> 16;
        col = q - ui * p.m;
    };
    const int ub = p.batch / p.subs;  // units per batch
    // The first output of this thread may add a residual value or be addressed by a position that earlier kernels
    // wrote: both are fetched now, beside the dot products.
    __half res_first = __ushort_as_half((unsigned short)0);
    int pos_first = 0;
    bool have_first = false;
    if (ks == 1) {
        int ui, col;
        split_q(tid >> 4, ui, col);
        if (ui < min(ub, n_mine)) {
            int ti, sl;
            place(unit_at(ui), ti, sl);
            const int n = sl * kRows + row16;
            if (n < p.t[ti].n) {
                have_first = true;
                pos_first = p.positions ? p.positions[col] : p.pos_offset + col;
                if (p.epilogue == TLC_EPI_RESIDUAL) res_first = p.residual[(size_t)col * p.t[ti].n + n];
            }
        }
    }

    // One output from its f32 sums: `v` of row n, `vp` of row n ^ 1 (RoPE), `vu` of the up projection.
    auto store_out = [&](int ti, int n, int col, float v, float vp, float vu, bool first) {
        const GemvTensor &o = p.t[ti];
        __half h = __float2half_rn(v);
        const size_t oidx = (size_t)col * o.n + n;  // dense [m, N] index (residual, act)
        int pos = first ? pos_first : p.positions ? p.positions[col] : p.pos_offset + col;
        // Second line of defence behind the host-side bound of the positions: a position outside the cache is
        // brought back to its last row, so the store stays inside the allocation; the attention kernel of
        // the same layer meets the same position, cuts it and raises the status word (TLC_ERR_INDEX).
        if (p.max_pos > 0) pos = min(max(pos, 0), p.max_pos - 1);
        // Dense rows by default; a KV-cache destination addresses rows by (sequence, position).
        __half *y = o.y + (size_t)((long long)col * o.row_stride + (long long)pos * o.pos_stride) + n;
        if (o.rope_heads > 0) {
            // interleaved RoPE on the f16-rounded projection (rope_f16, shaders/unified.metal:2355-2417)
            const __half hp = __float2half_rn(vp);
            const int dim = n % o.head_dim, pair = dim >> 1;
            const float x0 = __half2float((dim & 1) ? hp : h), x1 = __half2float((dim & 1) ? h : hp);
            const float freq = 1.0f / powf(p.rope_base, (float)(2 * pair) / (float)o.head_dim);
            const float theta = (float)(unsigned)pos * freq;
            const float cs = cosf(theta), sn = sinf(theta);
            *y = __float2half_rn((dim & 1) ? __fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, cs))
                                           : __fsub_rn(__fmul_rn(x0, cs), __fmul_rn(x1, sn)));
        } else if (p.epilogue == TLC_EPI_RESIDUAL) {
            *y = __hadd(h, first ? res_first : p.residual[oidx]);
        } else if (p.epilogue == TLC_EPI_SWIGLU) {
            // h = gate; s = sigmoid(g) (f32, RNE); a = g*s; act = a*u: three f16 roundings as in
            // debug/chat_demo_with_kvcache.tl:26-41
            const __half sg = __float2half_rn(1.0f / (1.0f + expf(-__half2float(h))));
            p.t[0].y[oidx] = __hmul(__hmul(h, sg), __float2half_rn(vu));
        } else {
            if (p.bias) h = __hadd(h, p.bias[n]);
            *y = h;
        }
    };

    // (b) main loop: slabs in batches of p.batch, one cross-warp reduction per batch
    int rs = 0;
    uint32_t rpar = 0;
    const uint32_t warp_off = (uint32_t)(wt0 * TILE);
    int slab = 0;  // of this CTA
    uint32_t epar = 0;
    const int round_units = ks > 1 ? p.round / p.subs : max(n_mine, 1);  // cluster: units between two exchanges
    for (int r0 = 0, batch_count = 0; r0 < n_mine || (ks > 1 && r0 < p.n_rounds * round_units); r0 += round_units) {
        const int r1 = min(n_mine, r0 + round_units);
        for (int i0 = r0; i0 < r1; i0 += ub, batch_count++) {
            const int nsets = min(ub, r1 - i0) * p.subs;
            float *rbuf = red + (size_t)(batch_count & 1) * p.batch * lay.red_slot;
            for (int a = 0; a < nsets; a++) {
                float acc[4 * NT];
#pragma unroll
                for (int i = 0; i < 4 * NT; i++) acc[i] = 0.f;
                // Refill the stage of the slab before, when all warps have read it.
                if (slab > 0 && (slab - 1) % CW == warp && slab - 1 + S < n_slabs) {
                    const int ps = rs == 0 ? S - 1 : rs - 1;
                    if (warp_wait(&empty[ps], epar, abort_flag, p.status, 1, p.wait_ns) && lane == 0) fetch(slab - 1 + S, ps);
                }
                if (rs == 0 && slab > 0) epar ^= 1u;  // (the stage before the first is the last one of the round before)
                // A wait that ran out skips the math but keeps the barrier protocol going.
                const bool ready = n_slabs > 0 && warp_wait(&full[rs], rpar, abort_flag, p.status, 2, p.wait_ns);
                const uint32_t sb = ring + (uint32_t)(rs * p.stage_bytes) + warp_off;
                const int nt_tiles = ready ? my_tiles : 0;
                if constexpr (Q6) {
                    if (nt_tiles > 0) {
                        // Super-block of the warp, rows g and g + 8: 128 low nibbles pairs, 64 high bit quads, 16 scales, d
                        // (GGUFLoader::dequantize_q6_k, src/model/formats/gguf.rs:128-218).  The word of lane t holds
                        // elements 4t .. 4t+3 of four groups of 16, 32 apart; a 6-bit value in the low bits of
                        // a binary16 is the subnormal q * 2^-24, the -32 is in the start value, and the group's 8-bit
                        // scale multiplies the 16 x 8 result in f32, the super-block's d at the end.
                        const uint32_t r0 = ring + (uint32_t)(rs * p.stage_bytes) + (uint32_t)((warp >> 3) * kQ6Box + (warp & 7) * 224) + g * kQ6BoxRow;
                        const uint32_t r1 = r0 + 8 * kQ6BoxRow;
                        float part0[2 * NT], part1[2 * NT];
#pragma unroll
                        for (int i = 0; i < 2 * NT; i++) part0[i] = part1[i] = 0.f;
                        const uint4 s0 = lds_u128(r0 + 192), s1 = lds_u128(r1 + 192);
                        const uint32_t sw0[4] = {s0.x, s0.y, s0.z, s0.w}, sw1[4] = {s1.x, s1.y, s1.z, s1.w};
                        const __half2 m1152 = __float2half2_rn(-1152.f);
                        // signed byte i of a scale word pair -> float, two at a time (1024 + 128 + sc, minus 1152: exact)
                        auto scales2 = [&](uint32_t w, int hi) {
                            const uint32_t h = __byte_perm(w ^ 0x80808080u, 0x64646464u, hi ? 0x4342 : 0x4140);
                            return __half22float2(__hadd2(*reinterpret_cast<const __half2 *>(&h), m1152));
                        };
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            // group j (elements 32 j + 16 is + ...) of half h has scale 8 h + is + 2 j
                            float2 sc0[4], sc1[4];
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                sc0[j] = scales2(sw0[2 * h + (j >> 1)], j & 1);
                                sc1[j] = scales2(sw1[2 * h + (j >> 1)], j & 1);
                            }
#pragma unroll
                            for (int is = 0; is < 2; is++) {
                                const uint32_t o = (uint32_t)(64 * h + 16 * is + 4 * t), oh = (uint32_t)(128 + 32 * h + 16 * is + 4 * t);
                                const uint32_t qa[2] = {lds_u32(r0 + o), lds_u32(r1 + o)}, qb[2] = {lds_u32(r0 + o + 32), lds_u32(r1 + o + 32)};
                                const uint32_t qh[2] = {lds_u32(r0 + oh), lds_u32(r1 + oh)};
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    uint32_t a[4];
#pragma unroll
                                    for (int r = 0; r < 2; r++) {
                                        const uint32_t lo4 = (j & 1 ? qb[r] : qa[r]) >> (j >= 2 ? 4 : 0);
                                        const uint32_t hi2 = j == 0 ? qh[r] << 4 : j == 1 ? qh[r] << 2 : j == 2 ? qh[r] : qh[r] >> 2;
                                        const uint32_t v = (lo4 & 0x0F0F0F0Fu) | (hi2 & 0x30303030u);
                                        a[r] = __byte_perm(v, 0, 0x4140);
                                        a[2 + r] = __byte_perm(v, 0, 0x4342);
                                    }
                                    const int b = 8 * h + 2 * j + is;  // group of the super-block: elements 128 h + 32 j + 16 is
                                    const float e0 = is ? sc0[j].y : sc0[j].x, e1 = is ? sc1[j].y : sc1[j].x;
#pragma unroll
                                    for (int nt = 0; nt < NT; nt++) {
                                        const float2 ci = lds_f32x2(ci_addr + (uint32_t)((b * MP + nt * 8) * 4));
                                        const float cc[4] = {ci.x, ci.y, ci.x, ci.y};
                                        float d[4];
                                        mma16816(d, a, xb[nt][b][0], xb[nt][b][1], cc);
                                        part0[2 * nt] = fmaf(e0, d[0], part0[2 * nt]);
                                        part0[2 * nt + 1] = fmaf(e0, d[1], part0[2 * nt + 1]);
                                        part1[2 * nt] = fmaf(e1, d[2], part1[2 * nt]);
                                        part1[2 * nt + 1] = fmaf(e1, d[3], part1[2 * nt + 1]);
                                    }
                                }
                            }
                        }
                        const float d0 = __half2float(__ushort_as_half((unsigned short)lds_u32(r0 + 208)));
                        const float d1 = __half2float(__ushort_as_half((unsigned short)lds_u32(r1 + 208)));
#pragma unroll
                        for (int nt = 0; nt < NT; nt++) {
                            acc[nt * 4 + 0] = d0 * part0[2 * nt];
                            acc[nt * 4 + 1] = d0 * part0[2 * nt + 1];
                            acc[nt * 4 + 2] = d1 * part1[2 * nt];
                            acc[nt * 4 + 3] = d1 * part1[2 * nt + 1];
                        }
                    }
                } else {
#pragma unroll
                for (int i = 0; i < TW; i++) {
                    if (i >= nt_tiles) break;
                    // words and scales of one tile for this lane: rows g (lo) and g + 8 (hi)
                    const uint32_t tb = sb + (uint32_t)i * TILE;
                    const uint4 vlo = lds_u128(tb + lane * 16), vhi = lds_u128(tb + 512 + lane * 16);
                    const uint32_t lo[4] = {vlo.x, vlo.y, vlo.z, vlo.w}, hi[4] = {vhi.x, vhi.y, vhi.z, vhi.w};
                    uint32_t slo[2], shi[2];
                    if (QT == TLC_TYPE_Q4_0) {
                        const uint2 x = lds_u64(tb + 1024 + g * 8), y = lds_u64(tb + 1024 + (g + 8) * 8);
                        slo[0] = x.x; slo[1] = x.y;
                        shi[0] = y.x; shi[1] = y.y;
                    } else {
                        slo[0] = lds_u32(tb + 1024 + g * 4);
                        shi[0] = lds_u32(tb + 1024 + (g + 8) * 4);
                        slo[1] = shi[1] = 0;
                    }
                    float dlo[4], dhi[4];
#pragma unroll
                    for (int h = 0; h < T::TB / 2; h++) {
                        const float2 l = __half22float2(*reinterpret_cast<const __half2 *>(&slo[h]));
                        const float2 u = __half22float2(*reinterpret_cast<const __half2 *>(&shi[h]));
                        dlo[2 * h] = l.x; dlo[2 * h + 1] = l.y;
                        dhi[2 * h] = u.x; dhi[2 * h + 1] = u.y;
                    }
#pragma unroll
                    for (int j = 0; j < T::TB; j++) {
                        const int b = i * T::TB + j;
                        uint32_t w0[2], w1[2], a1[4], a2[4];
                        if (QT == TLC_TYPE_Q4_0) {
                            w0[0] = lo[j];
                            w1[0] = hi[j];
                            w0[1] = w1[1] = 0;
                        } else {
                            w0[0] = lo[2 * j];
                            w0[1] = lo[2 * j + 1];
                            w1[0] = hi[2 * j];
                            w1[1] = hi[2 * j + 1];
                        }
                        unpack<QT>(w0, w1, a1, a2);
#pragma unroll
                        for (int nt = 0; nt < NT; nt++) {
                            const float2 ci = lds_f32x2(ci_addr + (uint32_t)((b * MP + nt * 8) * 4));
                            const float cc[4] = {ci.x, ci.y, ci.x, ci.y};
                            float d1[4], d2[4];
                            mma16816(d1, a1, xb[nt][b][0], xb[nt][b][1], cc);
                            mma16816(d2, a2, xb[nt][b][2], xb[nt][b][3], d1);
                            acc[nt * 4 + 0] = fmaf(dlo[j], d2[0], acc[nt * 4 + 0]);
                            acc[nt * 4 + 1] = fmaf(dlo[j], d2[1], acc[nt * 4 + 1]);
                            acc[nt * 4 + 2] = fmaf(dhi[j], d2[2], acc[nt * 4 + 2]);
                            acc[nt * 4 + 3] = fmaf(dhi[j], d2[3], acc[nt * 4 + 3]);
                        }
                    }
                }
                }
                __syncwarp();  // the stage has been read by all lanes
                if (lane == 0) mbar_arrive(&empty[rs]);
                slab++;
                if (++rs == S) {
                    rs = 0;
                    rpar ^= 1u;
                }
                float *mine = rbuf + a * lay.red_slot + warp * (MP * kRedPitch);
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    float *c = mine + (nt * 8 + 2 * t) * kRedPitch + g;
                    c[0] = acc[nt * 4 + 0];
                    c[kRedPitch] = acc[nt * 4 + 1];
                    c[8] = acc[nt * 4 + 2];
                    c[kRedPitch + 8] = acc[nt * 4 + 3];
                }
            }
            if (p.pdl_mode == 2 && i0 + ub >= n_mine) pdl_launch_dependents();
            consumer_bar<CT>();
            auto total = [&](int set, int row, int col) {
                const float *base = rbuf + set * lay.red_slot + col * kRedPitch + row;
                float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int w = 0; w < CW; w++) v[w & 3] += base[w * (MP * kRedPitch)];
                return (v[0] + v[1]) + (v[2] + v[3]);
            };
            if (ks > 1) {
                // this CTA's share of the sums: [set of the round][activation row][16]
                for (int q = tid >> 4; q < nsets * p.m; q += CT / 16) {
                    int set, col;
                    split_q(q, set, col);
                    part[(((i0 - r0) * p.subs + set) * MP + col) * 16 + row16] = total(set, row16, col);
                }
                continue;
            }
            for (int q = tid >> 4; q < (nsets >> (p.subs - 1)) * p.m; q += CT / 16) {  // subs is 1 or 2
                int ui, col, ti, sl;
                split_q(q, ui, col);
                place(unit_at(i0 + ui), ti, sl);
                const int n = sl * kRows + row16;
                if (n >= p.t[ti].n) continue;
                constexpr float UP = 16777216.0f;  // undo the 2^-24 of the integer fragments
                const float v = total(ui * p.subs, row16, col) * UP;
                const float vp = p.t[ti].rope_heads > 0 ? total(ui, row16 ^ 1, col) * UP : 0.f;
                const float vu = p.subs == 2 ? total(ui * 2 + 1, row16, col) * UP : 0.f;
                store_out(ti, n, col, v, vp, vu, have_first && i0 == 0 && q == tid >> 4);
            }
        }
        if (ks > 1) {
            // The CTAs of the cluster take the round's outputs in turn and add the shares of all, in rank order.
            if (r0 == 0) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            const int nq = max(0, r1 - r0) * p.m, q_step = ks * (CT / 16);
            auto gather = [&](int set, int col, int rw) {
                const uint32_t at = smem_u32(part + ((size_t)set * MP + col) * 16 + rw);
                float v = 0.f;
                for (int q0 = 0; q0 < ks; q0 += 8) {
                    float s[8];
#pragma unroll
                    for (int q = 0; q < 8; q++) {  // in flight together
                        s[q] = 0.f;
                        if (q0 + q < ks) {
                            uint32_t ra;
                            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(at), "r"(q0 + q));
                            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(s[q]) : "r"(ra));
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 8; q++) v += s[q];
                }
                return v * 16777216.0f;
            };
            for (int q = rank * (CT / 16) + (tid >> 4); q < nq; q += 2 * q_step) {  // two outputs' loads in flight
                float v[2], vp[2], vu[2];
                int n[2], ti[2], col[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int qq = q + u * q_step;
                    int ui, sl;
                    split_q(qq < nq ? qq : q, ui, col[u]);
                    place(unit_at(r0 + ui), ti[u], sl);
                    n[u] = qq < nq ? sl * kRows + row16 : INT_MAX;
                    v[u] = gather(ui * p.subs, col[u], row16);
                    vp[u] = p.t[ti[u]].rope_heads > 0 ? gather(ui, col[u], row16 ^ 1) : 0.f;
                    vu[u] = p.subs == 2 ? gather(ui * 2 + 1, col[u], row16) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < 2; u++)
                    if (n[u] < p.t[ti[u]].n) store_out(ti[u], n[u], col[u], v[u], vp[u], vu[u], false);
            }
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    }
}

}  // namespace tlc_gemv
