// The fused dequant-GEMV kernel for one activation row (the decode step of one sequence).  See tlc_gemv.cu for
// the design notes, tlc_gemv_kernel.cuh for two and more rows.
//
// At this size a launch is a chain of latencies (previous kernel's drain, activations, first stage of the
// ring, cross-warp reduction, store); the row is read once, each thread keeping its pieces in registers
// across the block-wide sum of squares.
#pragma once

#include "tlc_gemv_common.cuh"

namespace tlc_gemv {

constexpr int kRow1HeaderBytes = 1024;  // mbarriers, abort flag, sum-of-squares partials

// Shared-memory layout (bytes from the start of dynamic shared memory):
//   0    full[12] mbarriers      128  empty[12] mbarriers      256  abort flag
//   512  sum-of-squares partials [consumer warps]
//   1024 red   [2][AS sets][consumer warps][16 rows] f32   cross-warp reduction, double buffered
//   ...  cinit [nblk_pad] float4, the accumulator start value of a block four times (a whole C fragment
//              in one load; columns past the first are never read back)
//   ...  xperm [nblk_pad][4 quad lanes] uint4    activations in fragment order
//   ...  ring  [stages][16 tiles]                weight tiles as they lie in HBM (128-byte aligned)
__host__ __device__ inline size_t row1_fixed_smem(int nblk_pad, int as, int cw = 8) {
    size_t s = kRow1HeaderBytes;
    s += (size_t)2 * as * cw * kRows * sizeof(float);
    s += (size_t)nblk_pad * sizeof(float4);
    s += (size_t)nblk_pad * 4 * sizeof(uint4);
    s += 128;  // ring alignment slack
    return s;
}

// Columns 1-7 of the 16x8 tensor-core tile are never read back, so every lane may load the same B fragments
// and accumulator start values: their shared-memory addresses are warp-uniform with compile-time strides.
// CW: consumer warps, 8 (two CTAs per SM) or 16 (one CTA per SM, for a K that leaves no room for two).
template <int QT, int AS, int CW>
__global__ void __launch_bounds__((CW + 1) * 32, CW == 8 ? 2 : 1) gemv_row1_kernel(const GemvParams p) {
    static_assert(CW == 8 || CW == 16, "8 or 16 consumer warps");
    constexpr int CT = CW * 32;  // consumer threads
    using T = QTraits<QT>;
    constexpr int TILE = T::TILE_BYTES;
    constexpr int STAGE_BYTES = kTilesPerStage * TILE;
    constexpr int KEEP = 4;  // pieces of the row a thread keeps

    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem);
    uint64_t *empty = reinterpret_cast<uint64_t *>(smem + 128);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 256);
    float *sq_part = reinterpret_cast<float *>(smem + 512);
    float *red = reinterpret_cast<float *>(smem + kRow1HeaderBytes);
    static_assert(kMaxStages * 8 <= 128 && 512 + CW * 4 <= kRow1HeaderBytes, "header layout");
    float4 *cinit = reinterpret_cast<float4 *>(red + 2 * AS * CW * kRows);
    uint4 *xperm = reinterpret_cast<uint4 *>(cinit + p.nblk_pad);
    uint8_t *stages = reinterpret_cast<uint8_t *>(xperm + (size_t)p.nblk_pad * 4);
    stages = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(stages) + 127) & ~(uintptr_t)127);

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int S = p.nstages;

    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CW);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    // The next kernel of the stream may be scheduled from here on: its producer
    // warps only read weights, everything else waits for this grid to finish.
    if (p.pdl_mode == 1) pdl_launch_dependents();

    // Units of this CTA.  Worked out here, before anything waits for the previous kernel: the divisions are
    // then off the critical path of the decode step.
    const int cta_i = blockIdx.x, cta_n = gridDim.x;
    const int u_lo = p.contig ? (int)((long long)cta_i * p.total_units / cta_n) : 0;
    const int u_hi = p.contig ? (int)((long long)(cta_i + 1) * p.total_units / cta_n) : 0;
    const int n_mine = p.contig ? u_hi - u_lo : ((int)p.total_units - cta_i + cta_n - 1) / cta_n;

    if (warp == CW) {
        // ------------------------------ producer ------------------------------
        // Weights are never written by a kernel, so the ring starts filling
        // before the previous kernel of the stream has finished.
        int rs = 0;
        uint32_t rpar = 1;
        const uint64_t policy = l2_evict_first_policy();
        for (int ui = 0; ui < n_mine; ui++) {
            const int unit = p.contig ? u_lo + ui : cta_i + ui * cta_n;
            for (int sub = 0; sub < p.subs; sub++) {
                int ti = 0, sl = unit;
                if (p.subs == 2) {
                    ti = sub;
                } else {
                    if (sl >= p.slabs[0]) { sl -= p.slabs[0]; ti = 1; }
                    if (ti == 1 && sl >= p.slabs[1]) { sl -= p.slabs[1]; ti = 2; }
                }
                const uint8_t *wbase = ti == 0 ? p.t[0].w : ti == 1 ? p.t[1].w : p.t[2].w;
                const size_t spitch = ti == 0 ? p.t[0].slab_pitch : ti == 1 ? p.t[1].slab_pitch : p.t[2].slab_pitch;
                for (int c = 0; c < p.nchunks; c++) {
                    const int s = rs;
                    // On a timeout the producer stops issuing copies; the consumers'
                    // own bounded waits then end the CTA.
                    if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], rpar, abort_flag, p.status, 1, p.wait_ns))) return;
                    if (++rs == S) {
                        rs = 0;
                        rpar ^= 1u;
                    }
                    // The stage's tiles are contiguous in HBM: one bulk copy.
                    const int ntiles = min(kTilesPerStage, p.ktiles - c * kTilesPerStage);
                    const uint32_t bytes = (uint32_t)(ntiles * TILE);
                    if (lane == 0) {
                        const uint8_t *src = wbase + (size_t)sl * spitch + (size_t)(c * kTilesPerStage) * TILE;
                        mbar_expect_tx(&full[s], bytes);
                        bulk_g2s_hint(stages + (size_t)s * STAGE_BYTES, src, bytes, &full[s], policy);
                    }
                }
            }
        }
        return;
    }

    // -------------------------------- consumers --------------------------------
    // The row goes into shared memory in fragment order: item = (block b, quad lane t).
    //   Q4_0 fragment order: {4t, 4t+2, 16+4t, 18+4t | 4t+1, 4t+3, 17+4t, 19+4t}
    //   Q8_0 fragment order: {8t .. 8t+7}
    const int ctid = tid;  // 0..CT-1
    const bool do_norm = p.norm_w != nullptr;
    const int items = p.nblk_pad * 4, live_items = p.nblk * 4;
    const int rounds = (items + CT - 1) / CT;
    auto piece = [&](const __half *row, int idx) {  // the item's eight values
        const __half *r = row + (idx >> 2) * 32;
        const int t = idx & 3;
        if (QT == TLC_TYPE_Q4_0) {
            const uint2 lo = *reinterpret_cast<const uint2 *>(r + 4 * t), hi = *reinterpret_cast<const uint2 *>(r + 16 + 4 * t);
            return make_uint4(lo.x, lo.y, hi.x, hi.y);
        }
        return *reinterpret_cast<const uint4 *>(r + 8 * t);
    };
    // The norm weights of a model do not come from the previous kernel: the first round's are fetched
    // (the later rounds' brought into the cache) while that kernel is still running.
    uint4 nw_first = make_uint4(0, 0, 0, 0);
    auto fetch_norm = [&]() {
        if (ctid < live_items) nw_first = piece(p.norm_w, ctid);
        for (int idx = ctid + CT; idx < live_items; idx += CT) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.norm_w + (idx >> 2) * 32));
    };
    if (do_norm && p.norm_early) fetch_norm();
    pdl_wait();  // the activations (and residual) come from the previous kernel
    // Mode 3: the successor may be scheduled while this CTA does its own work, but not before the
    // predecessor is done (its CTAs then never wait behind two grids).
    if (p.pdl_mode == 3) pdl_launch_dependents();

    uint4 xr[KEEP];
#pragma unroll
    for (int r = 0; r < KEEP; r++) {
        const int idx = ctid + r * CT;
        xr[r] = idx < live_items ? piece(p.x, idx) : make_uint4(0, 0, 0, 0);
    }
    float inv = 1.f;
    if (do_norm) {
        if (!p.norm_early) fetch_norm();
        float sq = 0.f;
        auto add = [&](const uint4 &v) {
            const __half2 *h = reinterpret_cast<const __half2 *>(&v);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __half22float2(h[j]);
                sq = fmaf(f.x, f.x, sq);
                sq = fmaf(f.y, f.y, sq);
            }
        };
#pragma unroll
        for (int r = 0; r < KEEP; r++) add(xr[r]);
        for (int idx = ctid + KEEP * CT; idx < live_items; idx += CT) add(piece(p.x, idx));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (lane == 0) sq_part[warp] = sq;
        consumer_bar<CT>();
        float ss = 0.f;
#pragma unroll
        for (int w = 0; w < CW; w++) ss += sq_part[w];
        inv = 1.0f / sqrtf(ss / (float)p.k + p.eps);
    }
    auto place_piece = [&](int r, const uint4 &raw4) {
        const int idx = ctid + r * CT;
        const bool live = idx < live_items;
        const __half *raw = reinterpret_cast<const __half *>(&raw4);
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; j++) f[j] = __half2float(raw[j]);
        if (do_norm && live) {
            const uint4 nw4 = r == 0 ? nw_first : piece(p.norm_w, idx);
            const __half *nw = reinterpret_cast<const __half *>(&nw4);
            // f16((x * inv) * w): two separately rounded f32 multiplies, then RNE
            // (Tensor::rms_norm_cpu, src/ops/normalization.rs:236-240).
#pragma unroll
            for (int j = 0; j < 8; j++)
                f[j] = __half2float(__float2half_rn(__fmul_rn(__fmul_rn(f[j], inv), __half2float(nw[j]))));
        }
        float v[8];
        if (QT == TLC_TYPE_Q4_0) {
            v[0] = f[0]; v[1] = f[2]; v[2] = f[4]; v[3] = f[6];
            v[4] = f[1]; v[5] = f[3]; v[6] = f[5]; v[7] = f[7];
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = f[j];
        }
        // the four items of a block are adjacent lanes: a 2-step shuffle gives the block sum
        float s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (idx < items) {
            __half2 o[4];  // exact: v[] are f16 values
#pragma unroll
            for (int j = 0; j < 4; j++) o[j] = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
            xperm[idx] = *reinterpret_cast<const uint4 *>(o);
            const float cv = -T::OFFSET * 5.9604644775390625e-08f * s;  // * 2^-24
            if ((idx & 3) == 0) cinit[idx >> 2] = make_float4(cv, cv, cv, cv);
        }
    };
#pragma unroll
    for (int r = 0; r < KEEP; r++)
        if (r < rounds) place_piece(r, xr[r]);
    for (int r = KEEP; r < rounds; r++) {
        const int idx = ctid + r * CT;
        place_piece(r, idx < live_items ? piece(p.x, idx) : make_uint4(0, 0, 0, 0));
    }
    consumer_bar<CT>();

    // main loop
    const int g = lane >> 2, t = lane & 3;
    const uint32_t xp_addr = smem_u32(xperm + t), ci_addr = smem_u32(cinit), stages_addr = smem_u32(stages);

    // Units of this CTA: with only a few per CTA a balanced contiguous range
    // (1.5 % faster on the TinyLlama decode step), otherwise blockIdx.x,
    // blockIdx.x + gridDim.x, ... so that neighbouring CTAs stream neighbouring
    // rows (9 % faster on a 132 MB weight).  They are processed in batches of AS
    // accumulator sets (one set = one 16-row slab; a gate/up unit takes two) with
    // ONE cross-warp reduction per batch.
    const int ub = AS >> (p.subs - 1);  // units per batch (subs is 1 or 2)
    // The first output of this thread (item `ctid` of the first batch) adds a residual value and / or
    // is addressed by a position that earlier kernels wrote: both are fetched now, so that their
    // latency runs beside the dot products instead of after the reduction at the very end of the
    // kernel (the tail of every kernel is on the critical path of a decode step).
    __half res_first = __ushort_as_half((unsigned short)0);
    int pos_first = 0;
    bool have_first = false;
    {
        const int ui = ctid >> 4, row = ctid & 15;
        if (ui < min(ub, n_mine)) {
            int ti = 0, sl = p.contig ? u_lo + ui : cta_i + ui * cta_n;
            if (p.subs == 1) {
                if (sl >= p.slabs[0]) { sl -= p.slabs[0]; ti = 1; }
                if (ti == 1 && sl >= p.slabs[1]) { sl -= p.slabs[1]; ti = 2; }
            }
            const int n = sl * kRows + row;
            const int wn = ti == 0 ? p.t[0].n : ti == 1 ? p.t[1].n : p.t[2].n;
            if (n < wn) {
                have_first = true;
                pos_first = p.positions ? p.positions[0] : p.pos_offset;
                if (p.epilogue == TLC_EPI_RESIDUAL) res_first = p.residual[n];
            }
        }
    }
    int rs = 0;           // ring position and its parity, carried from stage to stage
    uint32_t rpar = 0;
    int batch_count = 0;

    // Words and scales of one tile for this lane: rows g (lo) and g + 8 (hi).
    struct TileRegs {
        uint4 vlo, vhi;
        uint32_t slo[2], shi[2];
    };
    auto load_tile = [&](TileRegs &r, uint32_t tb) {
        r.vlo = lds_u128(tb + lane * 16);
        r.vhi = lds_u128(tb + 512 + lane * 16);
        if (QT == TLC_TYPE_Q4_0) {
            const uint2 a = lds_u64(tb + 1024 + g * 8), b = lds_u64(tb + 1024 + (g + 8) * 8);
            r.slo[0] = a.x; r.slo[1] = a.y;
            r.shi[0] = b.x; r.shi[1] = b.y;
        } else {
            r.slo[0] = lds_u32(tb + 1024 + g * 4);
            r.shi[0] = lds_u32(tb + 1024 + (g + 8) * 4);
            r.slo[1] = r.shi[1] = 0;
        }
    };

    for (int i0 = 0; i0 < n_mine; i0 += ub, batch_count++) {
        const int nsets = min(ub, n_mine - i0) * p.subs;
        float acc[AS][2];  // rows g and g + 8, column 0
#pragma unroll
        for (int a = 0; a < AS; a++)
            acc[a][0] = acc[a][1] = 0.f;

#pragma unroll
        for (int a = 0; a < AS; a++) {
            if (a >= nsets) break;
            // The math of one tile, block by block; B fragments and accumulator
            // start values of block j + 1 are fetched while block j is in the
            // tensor cores.  b0: first block of the tile.
            auto do_tile = [&](const TileRegs &r, uint32_t b0) {
                const uint32_t lo[4] = {r.vlo.x, r.vlo.y, r.vlo.z, r.vlo.w};
                const uint32_t hi[4] = {r.vhi.x, r.vhi.y, r.vhi.z, r.vhi.w};
                float dlo[4], dhi[4];
#pragma unroll
                for (int h = 0; h < T::TB / 2; h++) {
                    const float2 l = __half22float2(*reinterpret_cast<const __half2 *>(&r.slo[h]));
                    const float2 u = __half22float2(*reinterpret_cast<const __half2 *>(&r.shi[h]));
                    dlo[2 * h] = l.x; dlo[2 * h + 1] = l.y;
                    dhi[2 * h] = u.x; dhi[2 * h + 1] = u.y;
                }
                // B fragments 64 bytes and start values 16 bytes apart from block to block
                const uint32_t xa = xp_addr + b0 * 64u, ca = ci_addr + b0 * 16u;
                uint4 xp = lds_u128(xa);
                uint4 ci = lds_u128(ca);
#pragma unroll
                for (int j = 0; j < T::TB; j++) {
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
                    const uint4 xc = xp, cq = ci;
                    if (j + 1 < T::TB) {
                        xp = lds_u128(xa + (j + 1) * 64);
                        ci = lds_u128(ca + (j + 1) * 16);
                    }
                    const float cc[4] = {__uint_as_float(cq.x), __uint_as_float(cq.y), __uint_as_float(cq.z),
                                         __uint_as_float(cq.w)};
                    float d1[4], d2[4];
                    mma16816(d1, a1, xc.x, xc.y, cc);
                    mma16816(d2, a2, xc.z, xc.w, d1);
                    // only column 0 of the tile (d2[0], d2[2] of quad lane 0) is ever read back
                    acc[a][0] = fmaf(dlo[j], d2[0], acc[a][0]);
                    acc[a][1] = fmaf(dhi[j], d2[2], acc[a][1]);
                }
            };
            for (int c = 0; c < p.nchunks; c++) {
                // A wait that ran out skips the math but keeps the barrier protocol
                // going, so every warp still reaches the same bar.sync calls.
                const bool ready = __all_sync(0xffffffffu, mbar_wait(&full[rs], rpar, abort_flag, p.status, 2, p.wait_ns));
                const int ntiles = ready ? min(kTilesPerStage, p.ktiles - c * kTilesPerStage) : 0;
                const uint32_t sbase = stages_addr + (uint32_t)rs * STAGE_BYTES;
                const uint32_t cb0 = (uint32_t)(c * kTilesPerStage * T::TB);  // first block of the stage
                if (ntiles == kTilesPerStage) {
                    // Lane (g, t) reads the words of rows g and g + 8 of its warp's two tiles
                    // up front (four 16-byte loads), then runs the blocks.
                    constexpr int TPW = kTilesPerStage / CW;  // tiles per warp and stage
                    static_assert(TPW * CW == kTilesPerStage && TPW >= 1, "whole tiles per warp");
                    TileRegs r[TPW];
#pragma unroll
                    for (int i = 0; i < TPW; i++) load_tile(r[i], sbase + (uint32_t)(warp + i * CW) * TILE);
#pragma unroll
                    for (int i = 0; i < TPW; i++) do_tile(r[i], cb0 + (uint32_t)(warp + i * CW) * T::TB);
                } else {
                    for (int ti = warp; ti < ntiles; ti += CW) {
                        TileRegs r0;
                        load_tile(r0, sbase + (uint32_t)ti * TILE);
                        do_tile(r0, cb0 + (uint32_t)ti * T::TB);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[rs]);
                if (++rs == S) {
                    rs = 0;
                    rpar ^= 1u;
                }
            }
        }

        // cross-warp reduction and epilogue of the batch
        if (p.pdl_mode == 2 && i0 + ub >= n_mine) pdl_launch_dependents();
        float *rbuf = red + (size_t)(batch_count & 1) * (AS * CW * kRows);
        if (t == 0) {
#pragma unroll
            for (int a = 0; a < AS; a++) {
                if (a >= nsets) break;
                float *mine = rbuf + (a * CW + warp) * kRows;
                mine[g] = acc[a][0];
                mine[g + 8] = acc[a][1];
            }
        }
        consumer_bar<CT>();
        for (int item = ctid; item < (nsets >> (p.subs - 1)) * kRows; item += CT) {  // subs is 1 or 2
            const int ui = item >> 4, row = item & 15;
            const int a0 = ui * p.subs;
            int ti = 0, sl = p.contig ? u_lo + i0 + ui : cta_i + (i0 + ui) * cta_n;
            if (p.subs == 1) {
                if (sl >= p.slabs[0]) { sl -= p.slabs[0]; ti = 1; }
                if (ti == 1 && sl >= p.slabs[1]) { sl -= p.slabs[1]; ti = 2; }
            }
            const int n = sl * kRows + row;
            const int wn = ti == 0 ? p.t[0].n : ti == 1 ? p.t[1].n : p.t[2].n;
            if (n >= wn) continue;
            auto total = [&](int set, int r_) {
                const float *base = rbuf + (size_t)set * CW * kRows + r_;
                float v = 0.f;
#pragma unroll
                for (int w = 0; w < CW; w++) v += base[w * kRows];
                return v * 16777216.0f;  // undo the 2^-24 of the integer fragments
            };
            __half *yout = ti == 0 ? p.t[0].y : ti == 1 ? p.t[1].y : p.t[2].y;
            const long long pstride = ti == 0 ? p.t[0].pos_stride : ti == 1 ? p.t[1].pos_stride : p.t[2].pos_stride;
            const int rheads = ti == 0 ? p.t[0].rope_heads : ti == 1 ? p.t[1].rope_heads : p.t[2].rope_heads;
            const int hdim = ti == 0 ? p.t[0].head_dim : ti == 1 ? p.t[1].head_dim : p.t[2].head_dim;
            __half h = __float2half_rn(total(a0, row));
            const bool first = have_first && i0 == 0 && item == ctid;
            int pos = first ? pos_first : p.positions ? p.positions[0] : p.pos_offset;
            // Second line of defence behind the host-side bound of the positions: a position outside
            // the cache is brought back to its last row, so the store stays inside the allocation; the
            // attention kernel of the same layer meets the same position, cuts it and raises the status
            // word (TLC_ERR_INDEX).  A clamp, not a test: a branch with a status update in this loop
            // cost the TinyLlama decode step 1.5 %.
            if (p.max_pos > 0) pos = min(max(pos, 0), p.max_pos - 1);
            // Where this output goes: dense rows by default; a KV-cache destination
            // addresses rows by (sequence, position) instead.
            const size_t yidx = (size_t)((long long)pos * pstride) + n;
            if (rheads > 0) {
                // Interleaved RoPE on the f16-rounded projection
                // (rope_f16, shaders/unified.metal:2355-2417).
                const __half hp = __float2half_rn(total(a0, row ^ 1));
                const int dim = n % hdim;
                const int pair = dim >> 1;
                const float x0 = __half2float((dim & 1) ? hp : h);
                const float x1 = __half2float((dim & 1) ? h : hp);
                const float exponent = (float)(2 * pair) / (float)hdim;
                const float freq = 1.0f / powf(p.rope_base, exponent);
                const float theta = (float)(unsigned)pos * freq;
                const float cs = cosf(theta), sn = sinf(theta);
                const float r = (dim & 1) ? __fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, cs))
                                          : __fsub_rn(__fmul_rn(x0, cs), __fmul_rn(x1, sn));
                yout[yidx] = __float2half_rn(r);
            } else if (p.epilogue == TLC_EPI_RESIDUAL) {
                yout[yidx] = __hadd(h, first ? res_first : p.residual[n]);
            } else if (p.epilogue == TLC_EPI_SWIGLU) {
                // h = gate; s = sigmoid(g) (f32, RNE); a = g*s; act = a*u: three
                // f16 roundings as in debug/chat_demo_with_kvcache.tl:26-41.
                const __half up = __float2half_rn(total(a0 + 1, row));
                const float gf = __half2float(h);
                const __half sg = __float2half_rn(1.0f / (1.0f + expf(-gf)));
                const __half av = __hmul(h, sg);
                p.t[0].y[n] = __hmul(av, up);
            } else {
                if (p.bias) h = __hadd(h, p.bias[n]);
                yout[yidx] = h;
            }
        }
    }
}

}  // namespace tlc_gemv
