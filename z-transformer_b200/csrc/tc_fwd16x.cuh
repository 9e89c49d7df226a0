// attn_fwd_tc16x<D>: the f16-split forward for head widths above 128, on tiles of D = 192 or 256 columns.
//
// At 256 columns a head no longer fits the layout of attn_fwd_tc16 / tc16g: one O accumulator alone is 256 of
// the 512 TMEM columns, and a 64-key K or V tile (hi and lo planes) is 64 KB.  This kernel keeps their
// arithmetic (S = Qh.Kh + Qh.Kl + Ql.Kh on kind::f16, P scaled by 2^7 and split into f16 pairs written over S,
// O += Ph.Vh + Ph.Vl + Pl.Vh, online softmax in the log2 domain with a lazily moved maximum) and changes
// what the sizes force:
//   CTA    128 query rows of ONE head; 6 warps: four softmax warps (a thread per row, every key tile), TMA, MMA.
//   TMEM   [0, 128) Q hi as the A operand, [128, 128 + D) O, [384, 512) two S/P tiles of 64 columns.
//   smem   Q lo (an SS MMA for the Ql.Kh term), ONE K tile and ONE V tile, 64 KB each at D = 256.
//   K      is a ring of its 64-column blocks rather than of whole tiles: S contracts over the blocks one
//          after the other, a block is free as soon as its twelve MMAs have retired and the same block of the
//          next tile is fetched into it while the later blocks are still being read.  So S(j+1) can follow
//          S(j) at once although there is room for one K tile only.
//   MMA    S(0) S(1) | P.V(0) S(2) | P.V(1) S(3) | ...: the softmax of tile j+1 runs under P.V(j) and S(j+2).
//          V(j+1) is fetched 16 keys after 16 keys, each piece as soon as the MMAs of P.V(j) on the one before it have
//          retired: a tile took 5100 clocks with V fetched as a whole while S(j+2) ran, against 4000 of MMAs.
// With the rows leaving as bulk copies (below): us, batch 8, T 1024, 32/8 heads of 256 650 -> 594; one sequence of T 700, 8/2 heads
// of 160 41 -> 36; 2 sequences of T 4096, 32/8 of 256 1695 -> 1663.
// Per 64-key tile the tensor core issues 12 MMAs of N = 64 per block for S and 12 of N = D for P.V: heads of 132 to 192
// columns on a tile of 192 issue three quarters of what they cost padded to 256.
// The query tile lands as f32 in V's slot and where Q lo goes, and is split by the row threads; the rows leave through the K and V
// slots, a bulk copy a row.  Every wait is bounded; a wait that gives up raises g_tc_status.
//
// The backward at these widths: tc_bwd_wide.cuh.
#pragma once

#include "tc_fwd16.cuh"

namespace zt {
namespace tcf16 {

constexpr int kThreadsX = 6 * 32;

struct SharedX {
    uint64_t full_k[4], free_k[4], full_v[4], free_v[4];
    uint64_t a_ready, q_full, s_full[2], p_full[2], pv_done, staged, all_done;
    uint32_t tmem_base;
    volatile int abort;
};
__device__ __forceinline__ bool xwait(uint64_t *bar, uint32_t parity, SharedX *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}
__device__ __forceinline__ void xgive_up(SharedX *sh, int code) {
    sh->abort = code;
    atomicMax(&g_tc_status, code);
}

// kmap: K planes with a box of ONE 64-column block x 64 keys; vmap: V planes, the head's D / 64 blocks x 16 keys; qmap:
// Q planes, the head's blocks x 128 rows.
template <int D, bool FLUSH>
__global__ void __launch_bounds__(kThreadsX, 1)
    attn_fwd_tc16x(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                   const __grid_constant__ CUtensorMap qmap, const Params p) {
    constexpr int NB = D / 64, BN = 64;
    constexpr int KB = BN * 128;        // bytes of one 64-column block of one plane of a key tile (8 KB)
    constexpr int KP = NB * KB;         // one plane of a key tile (32 KB at 256 columns); a K or V tile is 2 KP
    constexpr int VB = NB * 16 * 128;   // one plane of 16 keys of a V tile (8 KB at 256 columns)
    constexpr int QB = 128 * 128;       // one block of the lo pieces of the 128-row query tile (16 KB)
    static_assert(QB == kQBlock && KP * 2 == NB * QB, "the f32 query tile fills V's slot and Q lo");
    constexpr int cQh = 0, cO = 128, cS0 = 384;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // K: block c of the tile at sK + c * 2 KB (hi, then lo); V: 16 keys c of the tile at sV + c * 2 VB (hi, then lo); Q lo: NB blocks
    uint8_t *sK = smem_raw, *sV = sK + 2 * KP, *sQl = sV + 2 * KP;
    SharedX *sh = reinterpret_cast<SharedX *>(sQl + NB * QB);

    const int warp = threadIdx.x >> 5;
    // launch order (x fastest): a head's query tiles, late (long) ones first
    // Small launches have every head of every sequence along x instead, tile by tile (see tile_by_tile).
    const int bx = p.by_tile ? (int)blockIdx.x / p.n_heads : 0;
    const int qt = p.by_tile ? (int)gridDim.y - 1 - (int)blockIdx.y : (int)gridDim.x - 1 - (int)blockIdx.x;
    const int h = p.by_tile ? (int)blockIdx.x - bx * p.n_heads : (int)blockIdx.y, bp = (int)blockIdx.z + bx;
    const int b = bp / p.parts, part = bp - b * p.parts;
    const int g = h / (p.n_heads / p.n_kv_heads);
    const int t0 = qt * 128;
    const int rows_end = (t0 + 128 < p.T) ? t0 + 128 : p.T;
    int n_tiles = (p.q_offset + rows_end + BN - 1) / BN, jb = 0;  // key tiles of this CTA, and the first of them
    if (p.parts > 1) {
        const int per = (n_tiles + p.parts - 1) / p.parts;
        jb = part * per;
        n_tiles = n_tiles - jb < per ? n_tiles - jb : per;
        if (n_tiles <= 0) {
            pdl_wait();
            pdl_launch();
            if (threadIdx.x < 128 && t0 + threadIdx.x < p.T)
                p.lse[part * p.lse_part + ((long long)b * p.T + t0 + threadIdx.x) * p.n_heads + h] = -INFINITY;
            return;  // (the whole CTA: nothing has been set up yet)
        }
    }
    const int B = p.batch;

    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; ++i) mbar_init(&sh->full_k[i], 1), mbar_init(&sh->free_k[i], 1);
        for (int i = 0; i < BN / 16; ++i) mbar_init(&sh->full_v[i], 1), mbar_init(&sh->free_v[i], 1);
        mbar_init(&sh->a_ready, 4);
        mbar_init(&sh->q_full, 1);
        for (int i = 0; i < 2; ++i) mbar_init(&sh->s_full[i], 1), mbar_init(&sh->p_full[i], 4);
        mbar_init(&sh->pv_done, 1);
        mbar_init(&sh->staged, 4);
        mbar_init(&sh->all_done, 1);
        sh->abort = (smem_u32(smem_raw) & 1023u) ? 60 : 0;
        if (sh->abort) atomicMax(&g_tc_status, 60);
        mbar_fence_init();
    }
    if (warp == 5) tmem_alloc(&sh->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    // (the query rows are older than the launch before this one, for whose planes and maxima pdl_wait() waits)

    if (warp == 4) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one() && !sh->abort) {
            tma_prefetch_desc(&qmap), tma_prefetch_desc(&kmap), tma_prefetch_desc(&vmap);
            // the query tile: the lower half of its columns in V's slot, the upper where Q lo goes
            mbar_arrive_expect_tx(&sh->q_full, 2 * NB * QB);
            load_q<D>(sV, &qmap, &sh->q_full, t0, h, b);
            pdl_wait();
            pdl_launch();
            int n_k = 0, n_v = 0;  // K blocks and V pieces issued
            bool live = true;
            auto load_k_block = [&](int j, int c) {
                if (j >= 1 && !xwait(&sh->free_k[c], (uint32_t)((j - 1) & 1), sh)) { xgive_up(sh, 61), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_k[c], 2 * KB);
                tma_load_4d(sK + c * 2 * KB, &kmap, &sh->full_k[c], 0, (jb + j) * BN, g * NB + c, b);
                tma_load_4d(sK + c * 2 * KB + KB, &kmap, &sh->full_k[c], 0, (jb + j) * BN, g * NB + c, B + b);
                ++n_k;
            };
            auto load_v = [&](int j) {
                for (int c = 0; c < BN / 16; ++c) {
                    if (j >= 1 && !xwait(&sh->free_v[c], (uint32_t)((j - 1) & 1), sh)) { xgive_up(sh, 61), live = false; return; }
                    mbar_arrive_expect_tx(&sh->full_v[c], 2 * VB);
                    tma_load_4d(sV + c * 2 * VB, &vmap, &sh->full_v[c], 0, (jb + j) * BN + c * 16, g * NB, b);
                    tma_load_4d(sV + c * 2 * VB + VB, &vmap, &sh->full_v[c], 0, (jb + j) * BN + c * 16, g * NB, B + b);
                    ++n_v;
                }
            };
            for (int c = 0; c < NB; ++c) load_k_block(0, c);
            if (!xwait(&sh->a_ready, 0, sh)) xgive_up(sh, 61), live = false;  // V's slot holds query columns until then
            if (live) load_v(0);
            for (int j = 1; live && j < n_tiles; ++j) {
                for (int c = 0; live && c < NB; ++c) load_k_block(j, c);
                if (live) load_v(j);
            }
            if (sh->abort) {
                // let the copies in flight land before the CTA's shared memory goes away
                mbar_wait(&sh->q_full, 0);
                for (int i = (n_k > NB ? n_k - NB : 0); i < n_k; ++i) mbar_wait(&sh->full_k[i % NB], (uint32_t)((i / NB) & 1));
                for (int i = (n_v > 4 ? n_v - 4 : 0); i < n_v; ++i) mbar_wait(&sh->full_v[i & 3], (uint32_t)((i >> 2) & 1));
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t id_s = idesc_f16(128, BN, false, false);
            const int steps = head_steps(p.dim_out);
            const uint32_t id_o = idesc_f16(128, 16 * steps, false, true);
            bool ok = xwait(&sh->a_ready, 0, sh);
            if (!ok) xgive_up(sh, 62);
            tc_fence_after();
            const uint32_t k_u32 = smem_u32(sK), v_u32 = smem_u32(sV), ql_u32 = smem_u32(sQl);
            // S(j) into buffer j & 1, block by block of the contraction
            auto issue_qk = [&](int j) -> bool {
                const uint32_t cS = cS0 + (j & 1) * BN;
#pragma unroll
                for (int c = 0; c < NB; ++c) {
                    if (!xwait(&sh->full_k[c], (uint32_t)(j & 1), sh)) return false;
                    tc_fence_after();
                    const uint64_t bkh = desc_kmajor(k_u32 + (uint32_t)(c * 2 * KB));
                    const uint64_t bkl = desc_kmajor(k_u32 + (uint32_t)(c * 2 * KB + KB));
                    const uint64_t bql = desc_kmajor(ql_u32 + (uint32_t)(c * QB));
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                        const int kk = c * 4 + ks;
                        if (kk >= steps) break;
                        const uint64_t dkh = desc_advance(bkh, ks * 32), dkl = desc_advance(bkl, ks * 32);
                        mma_ts_f16(tmem + cS, tmem + cQh + kk * 8, dkh, id_s, kk > 0);
                        mma_ts_f16(tmem + cS, tmem + cQh + kk * 8, dkl, id_s, 1);
                        mma_ss_f16(tmem + cS, desc_advance(bql, ks * 32), dkh, id_s, 1);
                    }
                    mma_commit(&sh->free_k[c]);
                }
                mma_commit(&sh->s_full[j & 1]);
                return true;
            };
            // P.V of tile j, 16 keys after 16 keys of the contraction
            auto issue_pv = [&](int j) -> bool {
                const bool fresh = j == 0 || (FLUSH && j % kFlushKeyTiles == 0);  // (O was flushed before tile j)
                const uint32_t cS = cS0 + (j & 1) * BN;
#pragma unroll
                for (int kk = 0; kk < BN / 16; ++kk) {
                    if (!xwait(&sh->full_v[kk], (uint32_t)(j & 1), sh)) return false;
                    tc_fence_after();
                    const uint32_t ac = (uint32_t)(32 * (kk >> 1) + (kk & 1) * 8);
                    const uint64_t dvh = desc_mnmajor_16b(v_u32 + (uint32_t)(kk * 2 * VB), 16 * 128);
                    const uint64_t dvl = desc_mnmajor_16b(v_u32 + (uint32_t)(kk * 2 * VB + VB), 16 * 128);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvh, id_o, (!fresh || kk > 0) ? 1 : 0);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvl, id_o, 1);
                    mma_ts_f16(tmem + cO, tmem + cS + ac + 16, dvh, id_o, 1);
                    mma_commit(&sh->free_v[kk]);
                }
                mma_commit(&sh->pv_done);
                return true;
            };
            if (ok && !issue_qk(0)) { xgive_up(sh, 63); ok = false; }
            if (ok && n_tiles > 1 && !issue_qk(1)) { xgive_up(sh, 63); ok = false; }
            for (int j = 0; ok && j < n_tiles; ++j) {
                if (!xwait(&sh->p_full[j & 1], (uint32_t)((j >> 1) & 1), sh)) {
                    xgive_up(sh, 64);
                    break;
                }
                tc_fence_after();
                if (!issue_pv(j)) { xgive_up(sh, 64); break; }
                if (j == n_tiles - 1) mma_commit(&sh->all_done);  // once, after the last P.V
                if (j + 2 < n_tiles && !issue_qk(j + 2)) { xgive_up(sh, 63); break; }  // over the P tile P.V(j) has just read
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ softmax rows: a thread per query row
        const int tid = threadIdx.x, lane = threadIdx.x & 31;
        const int t = t0 + tid, pos = p.q_offset + t;
        const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
        bool ok = true;
        float top = 0.f;  // max |q| of the row
        {
            // this thread's row: the hi pieces into TMEM, the lo ones where the upper columns were, which are in registers by then
            if (!__all_sync(0xffffffffu, xwait(&sh->q_full, 0, sh))) xgive_up(sh, 69), ok = false;
            if (p.rope && t < p.T) rotate_q(sV, tid, p.rope + (long long)t * (p.dim_out >> 1), p.dim_out >> 3, 0, p.dim_out >> 3);
            float4 upper[D / 8];
#pragma unroll
            for (int c = 0; c < D / 8; ++c) {
                upper[c] = *q_at(sV, tid, D / 8 + c);
                top = fmaxf(top, fmaxf(max_abs4(upper[c]), max_abs4(*q_at(sV, tid, c))));
            }
            const float mq = block_mult(__float_as_uint(top));
#pragma unroll
            for (int cb = 0; cb < D / 32; ++cb) {
                uint32_t qh[16], ql[16];
                if (cb < D / 64) split_q32([&](int c) { return *q_at(sV, tid, cb * 8 + c); }, mq, qh, ql);
                else split_q32([&](int c) { return upper[(cb - D / 64) * 8 + c]; }, mq, qh, ql);
                tmem_st16(tmem + lane_base + cQh + cb * 16, qh);
                store_q_piece(sQl, tid, cb, ql);
            }
            tmem_wait_st();
            fence_async_smem();
            tc_fence_before();
            mbar_arrive_warp(&sh->a_ready);
        }
        pdl_wait();
        const float mk = block_mult(p.amax_k[b * p.n_kv_heads + g]), mv = block_mult(p.amax_v[b * p.n_kv_heads + g]);
        publish_q_top(p, b * p.n_kv_heads + g, top);
        const float cs = score_scale(p.scale_log2, block_mult(__float_as_uint(top)), mk);
        float m_ref = -INFINITY, l = 0.f;
        float m_flushed = -INFINITY;  // the reference maximum of what has been flushed
        FlushRow row{};
        if (FLUSH) row = flush_row_at(p, p.out + part * p.out_part, b, t0 + warp * 32, h);
        for (int j = 0; ok && j < n_tiles; ++j) {
            if (!__all_sync(0xffffffffu, xwait(&sh->s_full[j & 1], (uint32_t)((j >> 1) & 1), sh))) {
                xgive_up(sh, 65);
                ok = false;
                break;
            }
            tc_fence_after();
            const int s0 = (jb + j) * BN;
            const uint32_t cS = cS0 + (j & 1) * BN;
            const bool diag = (s0 + BN - 1 > p.q_offset + t0 + warp * 32) && !ZT_DEFECT(1);
            uint32_t r0[32], r1[32];
            tmem_ld32_joined(tmem + lane_base + cS, r0);
            tmem_ld32_joined(tmem + lane_base + cS + 32, r1);
            tmem_wait_ld();
            if (diag) mask32(r0, pos - s0), mask32(r1, pos - s0 - 32);
            const float mt = row_max32(r1, row_max32(r0, -INFINITY)) * cs;  // cs > 0
            float factor = 1.f;
            const float m_old = m_ref;
            if ((mt > m_ref + kRescaleThreshold || m_ref == -INFINITY) && mt != -INFINITY) {
                factor = (m_ref == -INFINITY) ? 0.f : ex2(m_ref - mt);
                m_ref = mt;
            }
            if (ZT_DEFECT(3) && j > 0) factor = 1.f;
            l *= factor;
            const bool flush = FLUSH && j > 0 && j % kFlushKeyTiles == 0;
            const bool moved = __any_sync(0xffffffffu, factor != 1.f);
            if (j > 0 && (flush || moved)) {
                // O may only be touched once the previous P.V has retired
                if (!__all_sync(0xffffffffu, xwait(&sh->pv_done, (uint32_t)((j - 1) & 1), sh))) {
                    xgive_up(sh, 66);
                    ok = false;
                    break;
                }
                tc_fence_after();
                if (flush) {
                    const bool first = m_flushed == -INFINITY;
                    flush_row<D>(tmem + lane_base + cO, row, first ? 0.f : ex2(m_flushed - m_old), first);
                    m_flushed = m_old;
                    __syncwarp();  // (rows past the sequence were not summed)
                } else {
#pragma unroll 1
                    for (int c = 0; c < D; c += 32) {
                        uint32_t r[32];
                        tmem_ld32_joined(tmem + lane_base + cO + c, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * factor);
                        tmem_st32_joined(tmem + lane_base + cO + c, r);
                    }
                }
            }
            // l is kept in P's units (times kPScale), like O
            const float off = ((m_ref == -INFINITY) ? 0.f : m_ref) - 7.0f;  // log2 kPScale
            float psum;
            {
                uint32_t ph[16], pl[16];
                psum = row_exp32(r0, cs, off, ph, pl);
                tmem_st16_joined(tmem + lane_base + cS, ph);
                tmem_st16_joined(tmem + lane_base + cS + 16, pl);
                psum += row_exp32(r1, cs, off, ph, pl);
                tmem_st16_joined(tmem + lane_base + cS + 32, ph);
                tmem_st16_joined(tmem + lane_base + cS + 48, pl);
            }
            l += psum;
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive_warp(&sh->p_full[j & 1]);
        }
        if (ok && !__all_sync(0xffffffffu, xwait(&sh->all_done, 0, sh))) {
            xgive_up(sh, 68);
            ok = false;
        }
        // The rows go to global memory through shared memory (idle once all_done completes), each by its own thread as one bulk
        // copy: the stores of a warp that went through all rows, two instructions a row, took 7500 clocks.  (Rows 16 bytes
        // apart from a multiple of 128, so that eight threads' chunks lie in different banks.)  A row that goes to more
        // places than out goes by such stores all the same.
        constexpr int RS = D * 4 + 16;
        uint8_t *stage = smem_raw;
        const bool plain = p.o_planes == nullptr && p.out_peers.n == 0;
        if (ok) {
            tc_fence_after();
            const float inv = l == 0.f ? 0.f : 1.f / (l * mv);  // l, like O, carries kPScale (0: a part without a key the row sees)
            const bool add = FLUSH && m_flushed != -INFINITY && row.sums != nullptr;
            const float ff = add ? ex2(m_flushed - m_ref) : 0.f;
            uint8_t *srow = stage + tid * RS;
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                uint32_t ra[32];
                tmem_ld32(tmem + lane_base + cO + c, ra);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    float4 o4 = make_float4(__uint_as_float(ra[i]), __uint_as_float(ra[i + 1]), __uint_as_float(ra[i + 2]), __uint_as_float(ra[i + 3]));
                    if (add && c + i < row.width) o4 = flush_sum4(row.at(c + i), ff, false, o4);
                    o4.x *= inv, o4.y *= inv, o4.z *= inv, o4.w *= inv;
                    *reinterpret_cast<float4 *>(srow + (c + i) * 4) = o4;
                }
            }
            if (p.lse && t < p.T) p.lse[part * p.lse_part + ((long long)b * p.T + t) * p.n_heads + h] = (m_ref + log2f(l) - 7.0f) * kLn2;
        }
        if (plain) send_row<FLUSH>(p.out + part * p.out_part + (((long long)b * p.T + t) * p.n_heads + h) * p.dim_out, stage + tid * RS, p.dim_out, ok && t < p.T);
        mbar_arrive_warp(&sh->staged);
        if (!plain && __all_sync(0xffffffffu, xwait(&sh->staged, 0, sh)) && !sh->abort) {
            const long long wo = (long long)p.n_heads * p.dim_out;
            const float mo = p.o_planes ? out_plane_mult(p, b) : 1.f;
            // a warp stores its 32 rows; a row is 48 or 64 chunks: two instructions
#pragma unroll 4
            for (int i = 0; i < 32; ++i) {
                const int r = warp * 32 + i;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int ch = half * 32 + lane;
                    if (ch >= D / 4) continue;
                    const float4 o4 = *reinterpret_cast<const float4 *>(stage + r * RS + ch * 16);
                    if (t0 + r < p.T && ch * 4 < p.dim_out)  // (a padded tile's upper columns are not the tensor's)
                        store_out4(p, part * p.out_part + ((long long)b * p.T + t0 + r) * wo + (long long)h * p.dim_out + ch * 4, o4, mo);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 5) tmem_dealloc(tmem, 512);
}

template <int D>
inline int launch_x_d(const CUtensorMap &kmap, const CUtensorMap &vmap, const CUtensorMap &qmap, const Params &p,
                    cudaStream_t stream) {
    const size_t smem = 3 * (size_t)(2 * 64 * D * 2) + sizeof(SharedX);  // K tile, V tile, Q lo
    const auto kernel = p.flush ? attn_fwd_tc16x<D, true> : attn_fwd_tc16x<D, false>;
    if (optin_smem((const void *)kernel, smem)) return 1;
    const dim3 grid = p.by_tile ? tile_major_grid(p.n_heads, (p.T + 127) / 128, p.batch * p.parts, kFwdTileWaves)
                                : dim3((unsigned)((p.T + 127) / 128), (unsigned)p.n_heads, (unsigned)(p.batch * p.parts));
    return launch_after("attn_fwd_tc16x", kernel, grid, dim3(kThreadsX), smem, stream, 1, kmap, vmap, qmap, p);
}

}  // namespace tcf16
}  // namespace zt
