// The one-kernel backward at tile width 64 (every head_dim up to 64, padded to it): tc_bwd_fused.cuh's protocol on steps of
// 128 query rows instead of 64.
//
// A head of 64 columns leaves half of what a 128-column head fills: with steps of 64 rows the row threads' hand-offs, not
// the tensor core, were what a step took (5500 clocks; the tensor pipe was active for 29 % of a launch at batch 8, T 512).  Here a step is a
// tile of 128 x 128 scores:
//  * S^T and dP^T are MMAs of N = 128, which cost 64 clocks where two of N = 64 cost 106, and a step's barriers,
//    polls and row constants serve twice the elements;
//  * dQ[t, d] = sum_s dS[t, s] K[s, d] has the step's 128 query rows as M (A = dS^T in shared memory read M-major, B = the
//    resident K tile N-major): a full tensor-core tile, where dQ^T had 64 rows of head columns and needed K's hi and lo
//    planes stacked on each other, twice the accumulator to drain;
//  * dQ, dK and dV leave by TMA (a reduction in memory), read out of TMEM by four warps of their own.  As
//    red.global.add.v4 the 32 KB of a step's dQ took 4300 clocks of an SM, 8 bytes a clock, and a flush of dK and dV 8000;
//  * the constants of a step's query rows are worked out by a warp of their own, a step ahead, and are three a row (a
//    broadcast LDS.128 is two wavefronts, and a step is bound by shared memory: 2500 wavefronts of loads and stores, 3200 of
//    the tensor core's operands and 770 of the copies', at 128 bytes a clock);
//  * the row threads' arithmetic is paired (fma.rn.f32x2).
// 16 row warps, a thread per key row and 32 of the step's query columns, at 80 registers a thread (all that 768 threads leave; the
// variants for split walks and padded heads spill 16 to 24 bytes).
// Sequences of up to 64 rows have half a step: ROWS = 64, a step of 128 x 64 scores, 16 query columns a row thread.  (Us, this kernel, steps
// of 128 -> of 64 rows: T 64, batch 64, 16/4 heads of 64 53.5 -> 45.5, one sequence of 16/16 heads of 32 14.8 -> 12.8; T 33, batch 256,
// 32/4 heads of 32 266 -> 208.  With T 129 to 192, whose second step is as empty, -10 to +10 %: those keep steps of 128.)
// TMEM: V hi 32 (of 64), S^T/P^T 128, dP^T/dS^T 128, dQ 64, dV 64, dK 64 = 512 columns.  Shared memory: K hi/lo, V lo 48 KB,
// dS^T hi/lo 64 KB, two Q slots and one dO slot of 32 KB each, 16 KB on the way out = 224 KB.
// Measured (us, before -> after, this kernel): 32/8 heads of 64, batch 8, T 512 139 -> 104, T 4096, batch 1 643 -> 448; heads
// of 32, batch 8, T 512 121 -> 94.  Error against 64 bits (2-norm, relative, N(0, 1); batch 2, T 512, 8/2 heads of 64): dq 8.0e-7 -> 5.8e-7, dk
// 9.2e-7 -> 6.9e-7, dv 7.3e-7 -> 6.2e-7.  (dQ sums three of the four products of the pieces where the kernel before it had all four: with
// lo.lo as well, 32 MMAs for 24, its error is the same to 1 %.  What moves it is dP's small terms going first; with its large ones
// first dq 7.2e-7.  Where the softmax is saturated on a few keys, dP and delta cancel and either order is within 9 % of the kernel before.)
#pragma once

#include "tc_bwd_wide.cuh"

namespace zt {
namespace tcf {

using namespace tc;
using namespace tcb;

struct Fused64Shared {
    uint64_t full_q[2], free_q[2], full_g, free_g;
    uint64_t k_full, a_ready, st_full, dp_full, p_ready, ds_ready, dq_done, dq_free, ld_ready, flush_ready, dv_free, dk_free;
    uint32_t tmem_base;
    volatile int abort;
    // per query row of the step: what turns K Q~^T into log2-domain scores, and minus the log-sum-exp; minus delta
    alignas(16) float csc[128], nlse[128], ndel[128];
};
__device__ __forceinline__ bool fwait(uint64_t *bar, uint32_t parity, Fused64Shared *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}
__device__ __forceinline__ void fgive_up(Fused64Shared *sh, int code) {
    sh->abort = code;
    atomicMax(&g_tc_status, code);
}

// The power of two at or below a normal x > 0; 0 for 0.
__device__ __forceinline__ float pow2_of(float x) { return __uint_as_float(__float_as_uint(x) & 0x7f800000u); }
// grid (n_kv_heads, ceil(T / 128), batch), 768 threads: 16 row warps, a TMA warp, two MMA warps, a warp for the rows'
// constants, four warps that read accumulators out.
constexpr int kFused64Threads = (kKvRowWarps + 8) * 32, kReadWarps = 4;
constexpr size_t kFused64Smem = 3 * (size_t)(128 * 64 * 2) + 2 * (size_t)(128 * 128 * 2) + 6 * (size_t)(128 * 64 * 2) +
                                kReadWarps * 4096 + sizeof(Fused64Shared);

// PARTS, PAD: as in attn_bwd_fused_tc.  ROWS: query rows of a step, 128, or 64 for sequences that have no more.
template <bool PARTS, bool PAD, int ROWS>
__global__ void __launch_bounds__(kFused64Threads, 1)
    attn_bwd_fused64_tc(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                        const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap gmap,
                        const __grid_constant__ CUtensorMap dqmap, const __grid_constant__ CUtensorMap dkmap,
                        const __grid_constant__ CUtensorMap dvmap, const BwdParams p) {
    constexpr int D = 64, BQ = ROWS, BR = 128 * 128;  // BR: bytes of 128 rows of 64 halves, every operand block's size
    constexpr int KP = BR, QP = BR, DSP = 2 * BR;    // one plane of K, of a query tile, of dS^T (two blocks of 64 query columns)
    const bool padded = PAD && plane_dim(p.dim_out) < D;  // the planes are narrower than the tile
    constexpr int cVh = 0, cST = 64, cDPT = 192, cDQ = 320, cDV = 384, cDK = 448;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *sKh = smem, *sKl = smem + KP, *sVl = smem + 2 * KP;  // V's hi plane sits in TMEM
    uint8_t *sDS = smem + 3 * KP;                                 // dS^T hi, lo: rows are keys
    uint8_t *sQ = sDS + 2 * DSP;                                  // slot s: Qh, Ql at sQ + s * 2 QP + {0, 1} QP
    uint8_t *sG = sQ + 2 * 2 * QP;                                // dOh, dOl
    uint8_t *sOut = sG + 2 * QP;                                  // 4 KB for each of the warps that read accumulators out
    Fused64Shared *sh = reinterpret_cast<Fused64Shared *>(sOut + kReadWarps * 4096);

    const int warp = threadIdx.x >> 5;
    // (the slowest index is the sequence, or the tile: see tile_by_tile)
    const int g = blockIdx.x, kt = PARTS && p.by_tile ? (int)blockIdx.z : (int)blockIdx.y, bp = PARTS && p.by_tile ? (int)blockIdx.y : (int)blockIdx.z;
    const int b = PARTS ? bp / p.parts.n() : bp, part = PARTS ? bp - b * p.parts.n() : 0;
    const int group = p.n_heads / p.n_kv_heads;
    const int s0 = kt * 128;
    // this CTA's part of the walk: heads [head0, head0 + n_heads_mine) and query tiles [qi0, n_q)
    const int n_heads_mine = PARTS ? group / p.parts.heads : group;
    const int head0 = PARTS ? g * group + part / p.parts.ranges * n_heads_mine : g * group;
    int n_q = (p.T + BQ - 1) / BQ, qi0 = kt * (128 / BQ);
    if (PARTS && p.parts.ranges > 1) {
        const int per = (n_q - qi0 + p.parts.ranges - 1) / p.parts.ranges;
        qi0 += part % p.parts.ranges * per;
        if (qi0 >= n_q) {
            pdl_wait();
            pdl_launch();
            return;  // (the whole CTA: nothing has been set up yet)
        }
        n_q = qi0 + per < n_q ? qi0 + per : n_q;
    }
    const int per_head = n_q - qi0;
    const int n_it = n_heads_mine * per_head;
    const int B = p.batch;
    WalkOf<BQ> walk(n_heads_mine, per_head, qi0, n_q);

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) mbar_init(&sh->full_q[i], 1), mbar_init(&sh->free_q[i], 1);
        mbar_init(&sh->full_g, 1), mbar_init(&sh->free_g, 2);  // (freed by two readers: dP^T and dV)
        mbar_init(&sh->k_full, 1);
        mbar_init(&sh->a_ready, kKvRowWarps);
        mbar_init(&sh->st_full, 1);
        mbar_init(&sh->dp_full, 1);
        mbar_init(&sh->p_ready, kKvRowWarps);
        mbar_init(&sh->ds_ready, kKvRowWarps);
        mbar_init(&sh->dq_done, 1);
        mbar_init(&sh->dq_free, BQ / 32);
        mbar_init(&sh->ld_ready, 1);
        mbar_init(&sh->flush_ready, 2);  // (dK's issuer and dV's)
        mbar_init(&sh->dv_free, kReadWarps), mbar_init(&sh->dk_free, kReadWarps);
        sh->abort = (smem_u32(smem) & 1023u) ? 70 : 0;
        if (sh->abort) atomicMax(&g_tc_status, 70);
        mbar_fence_init();
    }
    if (warp == kKvRowWarps + 1) tmem_alloc(&sh->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait();
    pdl_launch();

    const int bg = b * p.n_kv_heads + g;
    const float mq = block_mult(p.amax_q[bg]), mk = block_mult(p.amax_k[bg]);
    const float mv = block_mult(p.amax_v[bg]), mdo = block_mult(p.amax_do[bg]);
    const uint32_t rn_bits = p.dsmax[bg], vn_bits = p.vnmax[bg];  // (the header's last array holds max |dout row| here)
    const float cmin = ds_group_scale(rn_bits, vn_bits);
    // what turns K Q^T of the planes into log2-domain scores (where that is nothing -- q and k of 1e-12 -- something that still
    // is none to speak of: it is divided by)
    const float unit = fmaxf(p.scale_log2 / (mq * mk), 8.3e-25f);

    if (warp == kKvRowWarps) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one() && !sh->abort) {
            tma_prefetch_desc(&kmap), tma_prefetch_desc(&vmap), tma_prefetch_desc(&qmap), tma_prefetch_desc(&gmap);
            mbar_arrive_expect_tx(&sh->k_full, 3 * KP);
            load_head<1>(sKh, &kmap, &sh->k_full, s0, g, b, BR, padded);
            load_head<1>(sKl, &kmap, &sh->k_full, s0, g, B + b, BR, padded);
            load_head<1>(sVl, &vmap, &sh->k_full, s0, g, B + b, BR, padded);
            int n_ql = 0, n_gl = 0;  // tiles issued
            bool live = true;
            WalkOf<BQ> wq = walk, wg = walk;
            auto load_q = [&]() {  // Q tile of step n_ql
                const int j = n_ql, s = j & 1;
                // (its slot was last read by dK(j - 2))
                if (j >= 2 && !fwait(&sh->free_q[s], (uint32_t)((((j >> 1) - 1) & 1)), sh)) { fgive_up(sh, 71), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_q[s], 2 * BQ * 128);
                load_head<1>(sQ + s * 2 * QP, &qmap, &sh->full_q[s], wq.qi * BQ, head0 + wq.hh, b, BR, padded);
                load_head<1>(sQ + s * 2 * QP + QP, &qmap, &sh->full_q[s], wq.qi * BQ, head0 + wq.hh, B + b, BR, padded);
                ++n_ql, wq.next();
            };
            auto load_g = [&]() {  // dO tile of step n_gl
                const int j = n_gl;
                // (the one slot was last read by dV(j - 1) and dP^T(j - 1))
                if (j >= 1 && !fwait(&sh->free_g, (uint32_t)((j - 1) & 1), sh)) { fgive_up(sh, 71), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_g, 2 * BQ * 128);
                load_head<1>(sG, &gmap, &sh->full_g, wg.qi * BQ, head0 + wg.hh, b, BR, padded);
                load_head<1>(sG + QP, &gmap, &sh->full_g, wg.qi * BQ, head0 + wg.hh, B + b, BR, padded);
                ++n_gl, wg.next();
            };
            // the tensor core frees dO's slot (dV) before Q's (dK of the next step): ask in that order
            load_q(), load_g();
            if (n_it > 1) load_q();
            for (int it = 0; live && it < n_it; ++it) {
                if (it + 1 < n_it) load_g();
                if (live && it + 2 < n_it) load_q();
            }
            if (sh->abort) {
                // let the copies in flight land before the CTA's shared memory goes away
                mbar_wait(&sh->k_full, 0);
                for (int j = (n_ql > 2 ? n_ql - 2 : 0); j < n_ql; ++j) mbar_wait(&sh->full_q[j & 1], (uint32_t)((j >> 1) & 1));
                if (n_gl > 0) mbar_wait(&sh->full_g, (uint32_t)((n_gl - 1) & 1));
            }
        }
        __syncwarp();
    } else if (warp == kKvRowWarps + 1) {
        // ------------------------------------------------------------------ MMA issuer of the P side: S^T and dV (the split
        // between the two issuers, and why there are two, is attn_bwd_fused_tc's)
        if (elect_one()) {
            constexpr uint32_t id_s = idesc_f16(128, BQ, false, false);  // S^T: A = K, B = the query tile, both K-major
            const int steps = PAD ? head_steps(p.dim_out) : D / 16;
            const uint32_t id_a = idesc_f16(128, 16 * steps, false, true);  // dV: A in TMEM, B the dO tile N-major
            bool ok = !sh->abort && fwait(&sh->k_full, 0, sh);
            if (!ok) fgive_up(sh, 72);
            tc_fence_after();
            const uint64_t bkh = desc_kmajor(smem_u32(sKh)), bkl = desc_kmajor(smem_u32(sKl));
            const uint32_t q_u32 = smem_u32(sQ);
            const uint64_t mgh = desc_mnmajor_16b(smem_u32(sG), BR), mgl = desc_mnmajor_16b(smem_u32(sG) + QP, BR);
            auto wait_q = [&](int j) -> bool {
                if (!fwait(&sh->full_q[j & 1], (uint32_t)((j >> 1) & 1), sh)) return false;
                tc_fence_after();
                return true;
            };
            // S^T(j) = K Q~^T, its terms in the forward's order: the tensor core adds with truncation, and where the softmax is saturated
            // what dP and delta leave of each other is as good as this S agrees with the one that delta's P came from.  (Small terms
            // first here too: dq missed 1e-4 of its largest value by a quarter on scores that rise with the key, T 512, heads of 32.)
            auto issue_st = [&](int j) {
                const uint32_t qh = q_u32 + (uint32_t)((j & 1) * 2 * QP);
                const uint64_t bqh = desc_kmajor(qh), bql = desc_kmajor(qh + QP);
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    if (PAD && kk >= steps) break;
                    const uint64_t dkh = desc_advance(bkh, kk * 32), dqh = desc_advance(bqh, kk * 32);
                    mma_ss_f16(tmem + cST, dkh, dqh, id_s, kk > 0);
                    mma_ss_f16(tmem + cST, desc_advance(bkl, kk * 32), dqh, id_s, 1);
                    mma_ss_f16(tmem + cST, dkh, desc_advance(bql, kk * 32), id_s, 1);
                }
                mma_commit(&sh->st_full);
            };
            // dV(j) += P^T dO: P^T's 16-column windows hold hi halves in their first 8 columns, lo in the last 8.
            // Waits for P^T(j) and for dO(j); `restart`: the accumulators were flushed after step j-1.
            // (Here and in the other products the two small terms go first, while there is little to truncate.)
            int n_flush = 0;
            auto issue_dv = [&](int j, bool restart, bool flush_after) -> bool {
                if (!fwait(&sh->p_ready, (uint32_t)(j & 1), sh) || !fwait(&sh->full_g, (uint32_t)(j & 1), sh)) return false;
                if (restart && j > 0 && !fwait(&sh->dv_free, (uint32_t)((n_flush - 1) & 1), sh)) return false;
                tc_fence_after();
#pragma unroll
                for (int kk = BQ / 16 - 1; kk >= 0; --kk) {  // (late rows first, as the walk goes)
                    const uint64_t dgh = desc_advance(mgh, kk * 2048), dgl = desc_advance(mgl, kk * 2048);
                    mma_ts_f16(tmem + cDV, tmem + cST + kk * 16, dgl, id_a, (kk < BQ / 16 - 1 || !restart) ? 1u : 0u);
                    mma_ts_f16(tmem + cDV, tmem + cST + kk * 16 + 8, dgh, id_a, 1);
                    mma_ts_f16(tmem + cDV, tmem + cST + kk * 16, dgh, id_a, 1);
                }
                mma_commit(&sh->free_g);  // (one of two arrivals: the other issuer's dP^T(j) reads the same tile)
                if (flush_after) {
                    mma_commit(&sh->flush_ready);  // (one of two: the other issuer's dK(j))
                    ++n_flush;
                }
                return true;
            };
            // walk.* describe step `it`; step it+1's restart flag is step it's flush flag
            if (ok) {
                if (!wait_q(0)) { fgive_up(sh, 73); ok = false; }
                else {
                    issue_st(0);
                    if (!issue_dv(0, true, walk.flush)) { fgive_up(sh, 74); ok = false; }
                    else if (n_it > 1) {
                        if (!wait_q(1)) { fgive_up(sh, 73); ok = false; }
                        else issue_st(1);
                    }
                }
            }
            for (int it = 0; ok && it + 1 < n_it; ++it) {
                const bool restart = walk.flush;
                walk.next();  // now step it+1
                if (!issue_dv(it + 1, restart, walk.flush)) { fgive_up(sh, 74); break; }
                if (it + 2 < n_it) {
                    if (!wait_q(it + 2)) { fgive_up(sh, 73); break; }
                    issue_st(it + 2);
                }
            }
        }
        __syncwarp();
    } else if (warp == kKvRowWarps + 2) {
        // ------------------------------------------------------------------ MMA issuer of the dS side: dP^T, dK, dQ
        if (elect_one()) {
            constexpr uint32_t id_s = idesc_f16(128, BQ, false, false);  // dP^T: A = V (TMEM hi, shared lo), B = the dO tile K-major
            const int steps = PAD ? head_steps(p.dim_out) : D / 16;
            const uint32_t id_a = idesc_f16(128, 16 * steps, false, true);  // dK: A in TMEM, B the query tile N-major
            const uint32_t id_q = idesc_f16(128, 16 * steps, true, true);   // dQ: A = dS^T read M-major, B = K N-major
            bool ok = !sh->abort && fwait(&sh->k_full, 0, sh) && fwait(&sh->a_ready, 0, sh);
            if (!ok) fgive_up(sh, 72);
            tc_fence_after();
            const uint64_t bvl = desc_kmajor(smem_u32(sVl));
            const uint64_t bgh = desc_kmajor(smem_u32(sG)), bgl = desc_kmajor(smem_u32(sG) + QP);
            const uint64_t mkh = desc_mnmajor_16b(smem_u32(sKh), BR), mkl = desc_mnmajor_16b(smem_u32(sKl), BR);
            const uint64_t mdh = desc_mnmajor_16b(smem_u32(sDS), BR), mdl = desc_mnmajor_16b(smem_u32(sDS) + DSP, BR);
            const uint32_t q_u32 = smem_u32(sQ);
            // dP^T(j) = V dO^T (waits for dO(j))
            auto issue_dp = [&](int j) -> bool {
                if (!fwait(&sh->full_g, (uint32_t)(j & 1), sh)) return false;
                tc_fence_after();
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    if (PAD && kk >= steps) break;
                    mma_ts_f16(tmem + cDPT, tmem + cVh + kk * 8, desc_advance(bgl, kk * 32), id_s, kk > 0);
                    mma_ss_f16(tmem + cDPT, desc_advance(bvl, kk * 32), desc_advance(bgh, kk * 32), id_s, 1);
                }
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    if (PAD && kk >= steps) break;
                    mma_ts_f16(tmem + cDPT, tmem + cVh + kk * 8, desc_advance(bgh, kk * 32), id_s, 1);
                }
                mma_commit(&sh->free_g);  // (one of two arrivals: dV(j) reads the same tile)
                mma_commit(&sh->dp_full);
                return true;
            };
            // dQ(it): MMAs [first, first + 12) of the 24
            auto issue_dq = [&](int first) {
#pragma unroll
                for (int i = first; i < first + 12; ++i) {
                    const int kk = (i & 7) * 2048;
                    if (i < 8) mma_ss_f16(tmem + cDQ, desc_advance(mdl, kk), desc_advance(mkh, kk), id_q, i > 0);
                    else mma_ss_f16(tmem + cDQ, desc_advance(mdh, kk), desc_advance(i < 16 ? mkl : mkh, kk), id_q, 1);
                }
            };
            int n_flush = 0;
            if (ok && !issue_dp(0)) { fgive_up(sh, 73); ok = false; }
            for (int it = 0; ok && it < n_it; ++it, walk.next()) {
                if (!fwait(&sh->ds_ready, (uint32_t)(it & 1), sh)) { fgive_up(sh, 74); break; }
                // the accumulators restart at a step after a flush: they must have been read
                if (walk.fresh && it > 0 && !fwait(&sh->dk_free, (uint32_t)((n_flush - 1) & 1), sh)) { fgive_up(sh, 77); break; }
                tc_fence_after();
                {
                    // dK += dS^T Q~
                    const uint32_t qh = q_u32 + (uint32_t)((it & 1) * 2 * QP);
                    const uint64_t mqh = desc_mnmajor_16b(qh, BR), mql = desc_mnmajor_16b(qh + QP, BR);
                    const uint32_t acc0 = walk.fresh ? 0u : 1u;
#pragma unroll
                    for (int kk = BQ / 16 - 1; kk >= 0; --kk) {
                        const uint64_t dqh = desc_advance(mqh, kk * 2048), dql = desc_advance(mql, kk * 2048);
                        mma_ts_f16(tmem + cDK, tmem + cDPT + kk * 16, dql, id_a, kk < BQ / 16 - 1 ? 1u : acc0);
                        mma_ts_f16(tmem + cDK, tmem + cDPT + kk * 16 + 8, dqh, id_a, 1);
                        mma_ts_f16(tmem + cDK, tmem + cDPT + kk * 16, dqh, id_a, 1);
                    }
                    mma_commit(&sh->free_q[it & 1]);  // (S^T(it), the tile's other reader, retired before dS(it) could be formed)
                    if (walk.flush) {
                        mma_commit(&sh->flush_ready);  // (one of two: the other issuer's dV(it))
                        ++n_flush;
                    }
                }
                // dQ(it) over this CTA's 128 keys, in two halves with dP^T(it+1) between them, as in attn_bwd_fused_tc.
                // dQ's columns must have been read out first.
                if (it >= 1 && !fwait(&sh->dq_free, (uint32_t)((it - 1) & 1), sh)) { fgive_up(sh, 75); break; }
                tc_fence_after();
                issue_dq(0);
                if (it + 1 < n_it && !issue_dp(it + 1)) { fgive_up(sh, 73); break; }
                issue_dq(12);
                mma_commit(&sh->dq_done);  // dS^T(it) in shared memory has been read; dQ(it) can be read out
            }
        }
        __syncwarp();
    } else if (warp == kKvRowWarps + 3) {
        // ------------------------------------------------------------------ the constants of a step's query rows, four rows a
        // lane, fetched and worked out a step ahead.  (Done by the row threads, a value each, the loads' latency stood at the
        // head of every step and the arithmetic took a sixth of their instructions.)
        const int lane = threadIdx.x & 31;
        const float lse_shift = log2f(p.p_scale), ndel_unit = 1.0f / (p.p_scale * pow2_of(unit));
        constexpr int NR = BQ / 32;
        float lse[NR], rn[NR], de[NR];
        int t0 = walk.qi * BQ + lane;
        const auto load = [&]() {
            t0 = walk.qi * BQ + lane;
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const int t = t0 + i * 32;
                const long long idx = ((long long)b * p.T + (t < p.T ? t : 0)) * p.n_heads + head0 + walk.hh;
                // (the row sums may be the launch before's, pass_backward_kernel's: plain loads)
                lse[i] = __ldg(p.lse + idx), rn[i] = p.rnorm[idx], de[i] = p.delta[idx];
            }
        };
        load();
        for (int it = 0; it < n_it; ++it) {
            float csc[NR], nlse[NR], ndel[NR];
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const bool in = t0 + i * 32 < p.T;
                float cq, rel;
                ds_row_scale(rn[i], rn_bits, vn_bits, cq, rel);
                nlse[i] = in ? lse_shift - lse[i] * kLog2e : 0.f;
                ndel[i] = in && !ZT_DEFECT(13) ? -(de[i] * cmin * ndel_unit) : 0.f;
                csc[i] = in ? unit * (cq / cmin) : 0.f;
            }
            walk.next();
            if (it + 1 < n_it) load();
            // (every row warp has read the step before's)
            if (it > 0 && !__all_sync(0xffffffffu, fwait(&sh->ds_ready, (uint32_t)((it - 1) & 1), sh))) {
                fgive_up(sh, 68);
                break;
            }
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const int r = i * 32 + lane;
                sh->csc[r] = csc[i], sh->nlse[r] = nlse[i], sh->ndel[r] = ndel[i];
            }
            mbar_arrive_warp(&sh->ld_ready);
        }
    } else if (warp >= kKvRowWarps + 4) {
        // ------------------------------------------------------------------ what leaves TMEM for memory: dQ of every step, dV and
        // dK where they are flushed, by TMA through 4 KB of shared memory a warp: 32 rows x 32 columns, 128-byte swizzled.
        const int lane = threadIdx.x & 31, q32 = (warp & 3) * 32;
        const uint32_t lane_base = (uint32_t)q32 << 16;
        const float dq_unit = p.scale / mk;
        uint8_t *out = sOut + (warp & 3) * 4096;
        // columns [col, col + 32) of TMEM, this lane's row times f, into `out`
        const auto take = [&](uint32_t col, float f, uint64_t *freed) {
            uint32_t r[32];
            __syncwarp();  // (the whole warp: tcgen05.ld and its wait are warp-aligned)
            tmem_ld32(tmem + lane_base + col, r);
            if (lane == 0) tma_wait_read();
            __syncwarp();
            tmem_wait_ld();
            if (freed) {
                // (the tensor core may go on while the columns are still on their way)
                tc_fence_before();
                mbar_arrive_warp_relaxed(freed);
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float2 a = mul2(floats2(r[4 * c], r[4 * c + 1]), make_float2(f, f)), d = mul2(floats2(r[4 * c + 2], r[4 * c + 3]), make_float2(f, f));
                *reinterpret_cast<float4 *>(out + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_float4(a.x, a.y, d.x, d.y);
            }
            fence_async_smem();
            __syncwarp();
        };
        if (lane == 0) tma_prefetch_desc(&dqmap), tma_prefetch_desc(&dkmap), tma_prefetch_desc(&dvmap);
        const int bz = PARTS ? part * 2 * B + b : b;  // (the parts of dk and dv lie in turn)
        int n_flush = 0;
        for (int it = 0; it < n_it; ++it, walk.next()) {
            // this lane's query row of the step: 1 / (the scale of dS)
            const int t0 = walk.qi * BQ + q32;
            float fq = 0.f;
            if (q32 < BQ && t0 + lane < p.T) {
                float cq, rel;
                ds_row_scale(p.rnorm[((long long)b * p.T + t0 + lane) * p.n_heads + head0 + walk.hh], rn_bits, vn_bits, cq, rel);
                fq = dq_unit / cq;
            }
            if (walk.flush) {
                if (!__all_sync(0xffffffffu, fwait(&sh->flush_ready, (uint32_t)(n_flush & 1), sh))) {
                    fgive_up(sh, 76);
                    break;
                }
                tc_fence_after();
                if (lane == 0) tma_wait_done();  // (the flush before: sums are made in the order of the walk)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool is_dv = i < 2;
                    const int c0 = (i & 1) * 32;
                    take((is_dv ? cDV : cDK) + c0, is_dv ? 1.0f / (p.p_scale * mdo) : p.scale / (mq * cmin), i == 1 ? &sh->dv_free : i == 3 ? &sh->dk_free : nullptr);
                    if (lane == 0 && s0 + q32 < p.T && c0 < p.dim_out) {
                        const CUtensorMap *map = is_dv ? &dvmap : &dkmap;
                        if (n_flush == 0) tma_store_4d(map, out, c0, g, s0 + q32, bz);
                        else tma_add_4d(map, out, c0, g, s0 + q32, bz);
                        tma_commit();
                    }
                }
                ++n_flush;
            }
            if (q32 >= BQ) continue;  // (no query rows of the step)
            if (!__all_sync(0xffffffffu, fwait(&sh->dq_done, (uint32_t)(it & 1), sh))) {
                fgive_up(sh, 76);
                break;
            }
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < D; c0 += 32) {
                take(cDQ + c0, fq, c0 + 32 == D ? &sh->dq_free : nullptr);
                if (lane == 0 && t0 < p.T && c0 < p.dim_out) {
                    tma_add_4d(&dqmap, out, c0, head0 + walk.hh, t0, b);
                    tma_commit();
                }
            }
        }
        if (lane == 0) tma_wait_done();
    } else {
        // ------------------------------------------------------------------ one thread per key row and
        // 32 of the step's query columns: set `set` handles columns [32 set, 32 set + 32)
        constexpr int CW = BQ / 4;
        const int tid = threadIdx.x & 127, set = threadIdx.x >> 7;
        const int lane = threadIdx.x & 31;
        const int key = s0 + tid;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const int pd = PAD ? plane_dim(p.dim_out) : D;
        {
            // V's hi plane -> TMEM, 16 words of the row per set
            const long long off = ((long long)b * p.T + (key < p.T ? key : 0)) * p.n_kv_heads * pd + (long long)g * pd;
            if (set < 2) row_to_tmem16(p.v_planes + off + set * 32, key < p.T ? (pd - set * 32) / 8 : 0, tmem + lane_base + cVh + set * 16);
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive_warp(&sh->a_ready);
        }
        // dS = P (dP - delta) cq(t): the row threads keep P times csc(t)'s power of two, which beside cq(t) leaves with the units of
        // dP and delta.  (Powers of two only: dP and delta nearly cancel where the softmax is saturated, and a unit rounded once for
        // each of them left 1e-7 of delta there.)
        const float dp_unit = cmin / mdo / mv / (p.p_scale * pow2_of(unit));
        const float2 dp_unit2 = make_float2(dp_unit, dp_unit);
        float ds_top = 0.f;
        for (int it = 0; it < n_it; ++it, walk.next()) {
            const uint32_t par = (uint32_t)(it & 1);
            if (!__all_sync(0xffffffffu, fwait(&sh->ld_ready, par, sh) && fwait(&sh->st_full, par, sh))) {
                fgive_up(sh, 78);
                break;
            }
            tc_fence_after();
            const uint32_t wS = tmem + lane_base + cST + set * CW;
            const uint32_t wP = tmem + lane_base + cDPT + set * CW;
            float2 pr[CW / 2];
            {
                const float4 *csc = reinterpret_cast<const float4 *>(sh->csc + set * CW);
                const float4 *nlse = reinterpret_cast<const float4 *>(sh->nlse + set * CW);
                const int q_first = walk.qi * BQ, t0 = q_first + set * CW;
                const bool plain = (q_first >= s0 + 127 || ZT_DEFECT(11)) && q_first + BQ <= p.T && s0 + 128 <= p.T;
#pragma unroll
                for (int w = 0; w < CW / 16; ++w) {
                    uint32_t rs[16], ph[8], pl[8];
                    tmem_ld16(wS + 16 * w, rs);
                    tmem_wait_ld();
#pragma unroll
                    for (int i4 = 0; i4 < 4; ++i4) {
                        const float4 c = csc[4 * w + i4], n = nlse[4 * w + i4];
                        const int i = 4 * i4, k = 8 * w + 2 * i4;
                        const float2 x0 = fma2(floats2(rs[i], rs[i + 1]), make_float2(c.x, c.y), make_float2(n.x, n.y));
                        const float2 x1 = fma2(floats2(rs[i + 2], rs[i + 3]), make_float2(c.z, c.w), make_float2(n.z, n.w));
                        float2 p0 = make_float2(ex2(x0.x), ex2(x0.y)), p1 = make_float2(ex2(x1.x), ex2(x1.y));
                        if (!plain) {
                            const int t = t0 + 16 * w + i;
                            const auto vis = [&](int at) { return (key <= at || ZT_DEFECT(11)) && at < p.T && key < p.T; };
                            p0.x = vis(t) ? p0.x : 0.f, p0.y = vis(t + 1) ? p0.y : 0.f;
                            p1.x = vis(t + 2) ? p1.x : 0.f, p1.y = vis(t + 3) ? p1.y : 0.f;
                        }
                        pr[k] = mul2(p0, make_float2(pow2_of(c.x), pow2_of(c.y))), pr[k + 1] = mul2(p1, make_float2(pow2_of(c.z), pow2_of(c.w)));
                        split_pack(p0, ph[2 * i4], pl[2 * i4]);
                        split_pack(p1, ph[2 * i4 + 1], pl[2 * i4 + 1]);
                    }
                    tmem_st8(wS + 16 * w, ph);
                    tmem_st8(wS + 16 * w + 8, pl);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive_warp_relaxed(&sh->p_ready);
            if (!__all_sync(0xffffffffu, fwait(&sh->dp_full, par, sh))) {
                fgive_up(sh, 79);
                break;
            }
            tc_fence_after();
            bool free = true;
            {
                // The values go to the tensor core twice: over dP^T, and as a row of dQ's A operand -- key row `tid`, four 16-byte
                // chunks of its 128 bytes in the block of 64 query columns that they belong to, 128-byte swizzled.
                uint8_t *row_h = sDS + (set * CW >> 6) * BR + tid * 128;
                const float4 *ndel = reinterpret_cast<const float4 *>(sh->ndel + set * CW);
#pragma unroll
                for (int w = 0; w < CW / 16; ++w) {
                    uint32_t rd[16];
                    tmem_ld16(wP + 16 * w, rd);
                    tmem_wait_ld();
                    uint32_t th[8], tl[8];
#pragma unroll
                    for (int i4 = 0; i4 < 4; ++i4) {
                        const float4 n = ndel[4 * w + i4];
                        const int i = 4 * i4, k = 8 * w + 2 * i4;
                        float2 x0 = mul2(fma2(floats2(rd[i], rd[i + 1]), dp_unit2, make_float2(n.x, n.y)), pr[k]);
                        float2 x1 = mul2(fma2(floats2(rd[i + 2], rd[i + 3]), dp_unit2, make_float2(n.z, n.w)), pr[k + 1]);
                        x0.x = clamp_abs(x0.x, kDsBound), x0.y = clamp_abs(x0.y, kDsBound);
                        x1.x = clamp_abs(x1.x, kDsBound), x1.y = clamp_abs(x1.y, kDsBound);
                        ds_top = max3(max3(ds_top, fabsf(x0.x), fabsf(x0.y)), fabsf(x1.x), fabsf(x1.y));
                        split_pack(x0, th[2 * i4], tl[2 * i4]);
                        split_pack(x1, th[2 * i4 + 1], tl[2 * i4 + 1]);
                    }
                    tmem_st8(wP + 16 * w, th);
                    tmem_st8(wP + 16 * w + 8, tl);
                    // (dQ(it-1), issued around dP^T(it), may still be reading dS^T(it-1) there)
                    if (w == 0 && it >= 1) free = __all_sync(0xffffffffu, fwait(&sh->dq_done, (uint32_t)((it - 1) & 1), sh));
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int at = (((set * CW & 63) / 8 + 2 * w + c) ^ (tid & 7)) << 4;
                        *reinterpret_cast<uint4 *>(row_h + at) = make_uint4(th[4 * c], th[4 * c + 1], th[4 * c + 2], th[4 * c + 3]);
                        *reinterpret_cast<uint4 *>(row_h + DSP + at) = make_uint4(tl[4 * c], tl[4 * c + 1], tl[4 * c + 2], tl[4 * c + 3]);
                    }
                }
            }
            if (!free) {
                fgive_up(sh, 69);
                break;
            }
            tmem_wait_st();
            fence_async_smem();
            tc_fence_before();
            mbar_arrive_warp(&sh->ds_ready);
        }
        if (__any_sync(0xffffffffu, ds_top >= kDsBound) && lane == 0) atomicAdd(&g_tc_saturated, 1u);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kKvRowWarps + 1) tmem_dealloc(tmem, 512);
}

// Query rows of a step.  (One variant at 64 for whole and split walks, padded and whole heads.)
inline int fused64_rows(int T) { return T <= 64 ? 64 : 128; }

inline int launch_bwd_fused64(const CUtensorMap &k128, const CUtensorMap &v128, const CUtensorMap &qs128, const CUtensorMap &g128,
                              const BwdParams &p, cudaStream_t stream) {
    CUtensorMap dqmap, dkmap, dvmap;
    const long long kv_batch = p.parts.n() > 1 ? (2LL * p.parts.n() - 1) * p.batch : p.batch;
    if (!make_row_map(&dqmap, p.dq, p.batch, p.T, p.n_heads, p.dim_out, 32) ||
        !make_row_map(&dkmap, p.dk, kv_batch, p.T, p.n_kv_heads, p.dim_out, 32) ||
        !make_row_map(&dvmap, p.dv, kv_batch, p.T, p.n_kv_heads, p.dim_out, 32))
        return refuse("the TMA tensor maps for the backward's gradients could not be encoded.");
    const auto kernel = fused64_rows(p.T) == 64 ? attn_bwd_fused64_tc<true, true, 64>
                                  : with_flags([](auto parts, auto pad) { return attn_bwd_fused64_tc<parts.value, pad.value, 128>; }, p.parts.n() > 1 || p.by_tile, head_steps(p.dim_out) < 4);
    if (optin_smem((const void *)kernel, kFused64Smem)) return 1;
    const unsigned tiles = (unsigned)((p.T + 127) / 128), seqs = (unsigned)(p.batch * p.parts.n()), kv = (unsigned)p.n_kv_heads;
    const dim3 grid = p.by_tile ? dim3(kv, seqs, tiles) : dim3(kv, tiles, seqs);
    return launch_after("attn_bwd_fused64_tc", kernel, grid, dim3(kFused64Threads), kFused64Smem, stream, 1, k128, v128, qs128, g128, dqmap, dkmap, dvmap, p);
}

}  // namespace tcf
}  // namespace zt
