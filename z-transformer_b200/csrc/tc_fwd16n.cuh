// attn_fwd_tc16n: the f16-split forward of heads of up to 64 columns (narrower ones padded), two CTAs an SM.
//
// A tile of 64 keys is 768 clocks of MMAs here, half of what it is at 128 columns, while its softmax is as long as there: with one CTA
// an SM, two heads in it (attn_fwd_tc16g), a pair of tiles took 2700 clocks where the MMAs take 1660, and on the way to the first MMA
// and from the last one to memory (12000 clocks) nothing at all ran.  Two CTAs fill each other's gaps.  What makes room for the
// second:
//   CTA    128 query rows of ONE head; 6 warps: four softmax warps (a thread per row, every key tile), TMA, MMA.
//   TMEM   [0, 32) Q hi, [32, 64) Q lo, [64, 128) O, [128, 256) two S/P tiles of 64 columns: half of it.
//   smem   K ring and V ring of three slots each, 96 KB; the f32 query tile waits in V's first two slots, the rows leave through K's.
//   MMA    S(0) S(1) | P.V(0) S(2) | P.V(1) S(3) | ...: the softmax of tile j+1 runs under P.V(j) and S(j+2).
// The arithmetic is attn_fwd_tc16's (S's terms in the same order, one accumulator of O).
// Us of the kernel, the forms before (one or two heads a CTA, whichever took the call) -> this: batch 8, T 512, 32/8 heads 64 -> 48; 2 of T
// 3000, 16/16 heads 146 -> 93; 4 of 2000, 12/4 113 -> 70; 8 of 700, 12/4 54 -> 33; 8 of 4096, 32/8 1670 -> 1400; 16 of 130, 16/16 of 32
// columns 34 -> 21; 1500 rows at 4000 keys, 32/8 of 56 270 -> 197.  (Two heads a CTA, one CTA an SM, with two S buffers each and the
// next tiles' rows split ahead: 64 -> 54, 146 -> 121, 113 -> 87.)
#pragma once

#include "tc_fwd16.cuh"

namespace zt {
namespace tcf16 {

constexpr int kThreadsN = 6 * 32;

struct SharedN {
    uint64_t full_k[3], free_k[3], full_v[3], free_v[3];
    uint64_t a_ready, q_full, s_full[2], p_full[2], pv_done, staged, all_done;
    uint32_t tmem_base;
    volatile int abort;
};
__device__ __forceinline__ bool nwait(uint64_t *bar, uint32_t parity, SharedN *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}
__device__ __forceinline__ void ngive_up(SharedN *sh, int code) {
    sh->abort = code;
    atomicMax(&g_tc_status, code);
}

template <bool FLUSH, bool PAD>
__global__ void __launch_bounds__(kThreadsN, 2)
    attn_fwd_tc16n(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                   const __grid_constant__ CUtensorMap qmap, const Params p) {
    constexpr int D = 64, BN = 64;
    constexpr int KP = BN * D * 2;  // bytes of one plane of a key tile; a ring slot is 2 KP (hi, lo)
    constexpr int cQh = 0, cQl = 32, cO = 64, cS0 = 128;
    const bool padded = PAD && plane_dim(p.dim_out) < D;  // the planes are narrower than the tile
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *sK = smem_raw, *sV = sK + 6 * KP;
    SharedN *sh = reinterpret_cast<SharedN *>(sV + 6 * KP);

    const int warp = threadIdx.x >> 5;
    // launch order (x fastest): a head's query tiles, late (long) ones first, or every head of every sequence along x, tile by tile
    int qt, h, b;
    if (p.by_tile) {
        const int across = p.n_heads * p.batch;
        const int i = (int)blockIdx.x;
        const int r = i / across, u = i - r * across;
        qt = (p.T + 127) / 128 - 1 - r, b = u / p.n_heads, h = u - b * p.n_heads;
    } else {
        qt = (int)gridDim.x - 1 - (int)blockIdx.x, h = (int)blockIdx.y, b = (int)blockIdx.z;
    }
    const int g = h / (p.n_heads / p.n_kv_heads);
    const int t0 = qt * 128;
    const int rows_end = (t0 + 128 < p.T) ? t0 + 128 : p.T;
    const int n_tiles = (p.q_offset + rows_end + BN - 1) / BN;
    const int B = p.batch;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 3; ++i) {
            mbar_init(&sh->full_k[i], 1), mbar_init(&sh->free_k[i], 1);
            mbar_init(&sh->full_v[i], 1), mbar_init(&sh->free_v[i], 1);
        }
        mbar_init(&sh->a_ready, 4), mbar_init(&sh->q_full, 1);
        for (int i = 0; i < 2; ++i) mbar_init(&sh->s_full[i], 1), mbar_init(&sh->p_full[i], 4);
        mbar_init(&sh->pv_done, 1), mbar_init(&sh->staged, 4), mbar_init(&sh->all_done, 1);
        sh->abort = (smem_u32(smem_raw) & 1023u) ? 30 : 0;
        if (sh->abort) atomicMax(&g_tc_status, 30);
        mbar_fence_init();
    }
    if (warp == 5) tmem_alloc(&sh->tmem_base, 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    // (the query rows are older than the launch before this one, for whose planes and maxima pdl_wait() waits)

    if (warp == 4) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one() && !sh->abort) {
            tma_prefetch_desc(&qmap), tma_prefetch_desc(&kmap), tma_prefetch_desc(&vmap);
            mbar_arrive_expect_tx(&sh->q_full, 4 * KP);
            load_q<D>(sV, &qmap, &sh->q_full, t0, h, b);
            pdl_wait();
            pdl_launch();
            int n_k = 0, n_v = 0;  // tiles issued
            bool live = true;
            auto load_k = [&](int j) {
                const int s = j % 3;
                if (j >= 3 && !nwait(&sh->free_k[s], (uint32_t)(((j / 3) & 1) ^ 1), sh)) { ngive_up(sh, 31), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_k[s], 2 * KP);
                load_head<1>(sK + s * 2 * KP, &kmap, &sh->full_k[s], j * BN, g, b, BN * 128, padded);
                load_head<1>(sK + s * 2 * KP + KP, &kmap, &sh->full_k[s], j * BN, g, B + b, BN * 128, padded);
                ++n_k;
            };
            auto load_v = [&](int j) {
                const int s = j % 3;
                if (j >= 3 && !nwait(&sh->free_v[s], (uint32_t)(((j / 3) & 1) ^ 1), sh)) { ngive_up(sh, 31), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_v[s], 2 * KP);
                load_head<1>(sV + s * 2 * KP, &vmap, &sh->full_v[s], j * BN, g, b, BN * 128, padded);
                load_head<1>(sV + s * 2 * KP + KP, &vmap, &sh->full_v[s], j * BN, g, B + b, BN * 128, padded);
                ++n_v;
            };
            const int first = n_tiles < 3 ? n_tiles : 3;
            for (int j = 0; j < first; ++j) load_k(j);
            // V's slots are the query tile's until every row thread has read its row
            if (!nwait(&sh->a_ready, 0, sh)) ngive_up(sh, 31), live = false;
            for (int j = 0; live && j < first; ++j) load_v(j);
            for (int j = 3; live && j < n_tiles; ++j) {
                load_k(j);
                if (live) load_v(j);
            }
            if (sh->abort) {
                // let the copies in flight land before the CTA's shared memory goes away
                mbar_wait(&sh->q_full, 0);
                for (int j = (n_k > 3 ? n_k - 3 : 0); j < n_k; ++j) mbar_wait(&sh->full_k[j % 3], (uint32_t)((j / 3) & 1));
                for (int j = (n_v > 3 ? n_v - 3 : 0); j < n_v; ++j) mbar_wait(&sh->full_v[j % 3], (uint32_t)((j / 3) & 1));
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t id_s = idesc_f16(128, BN, false, false);
            const int steps = PAD ? head_steps(p.dim_out) : D / 16;
            const uint32_t id_o = idesc_f16(128, 16 * steps, false, true);
            bool ok = nwait(&sh->a_ready, 0, sh);
            if (!ok) ngive_up(sh, 32);
            tc_fence_after();
            const uint32_t k_u32 = smem_u32(sK), v_u32 = smem_u32(sV);
            // S of tile j into buffer j & 1
            auto issue_qk = [&](int j) -> bool {
                const int s = j % 3;
                if (!nwait(&sh->full_k[s], (uint32_t)((j / 3) & 1), sh)) return false;
                tc_fence_after();
                const uint32_t kh = k_u32 + (uint32_t)(s * 2 * KP);
                const uint64_t bkh = desc_kmajor(kh), bkl = desc_kmajor(kh + KP);
                const uint32_t cS = cS0 + (j & 1) * BN;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    if (PAD && kk >= steps) break;
                    const uint64_t dkh = desc_advance(bkh, kk * 32), dkl = desc_advance(bkl, kk * 32);
                    mma_ts_f16(tmem + cS, tmem + cQh + kk * 8, dkh, id_s, kk > 0);
                    mma_ts_f16(tmem + cS, tmem + cQh + kk * 8, dkl, id_s, 1);
                    mma_ts_f16(tmem + cS, tmem + cQl + kk * 8, dkh, id_s, 1);
                }
                mma_commit(&sh->free_k[s]);
                mma_commit(&sh->s_full[j & 1]);
                return true;
            };
            if (ok && !issue_qk(0)) { ngive_up(sh, 33); ok = false; }
            if (ok && n_tiles > 1 && !issue_qk(1)) { ngive_up(sh, 33); ok = false; }
            for (int j = 0; ok && j < n_tiles; ++j) {
                const int s = j % 3;
                if (!nwait(&sh->p_full[j & 1], (uint32_t)((j >> 1) & 1), sh) ||
                    !nwait(&sh->full_v[s], (uint32_t)((j / 3) & 1), sh)) { ngive_up(sh, 34); break; }
                tc_fence_after();
                const bool fresh = j == 0 || (FLUSH && j % kFlushKeyTiles == 0);  // (O was flushed before tile j)
                const uint32_t vh = v_u32 + (uint32_t)(s * 2 * KP);
                const uint64_t mvh = desc_mnmajor_16b(vh, BN * 128), mvl = desc_mnmajor_16b(vh + KP, BN * 128);
                const uint32_t cS = cS0 + (j & 1) * BN;
#pragma unroll
                for (int kk = 0; kk < BN / 16; ++kk) {
                    const uint32_t ac = (uint32_t)(32 * (kk >> 1) + (kk & 1) * 8);
                    const uint64_t dvh = desc_advance(mvh, kk * 2048), dvl = desc_advance(mvl, kk * 2048);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvh, id_o, (!fresh || kk > 0) ? 1 : 0);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvl, id_o, 1);
                    mma_ts_f16(tmem + cO, tmem + cS + ac + 16, dvh, id_o, 1);
                }
                mma_commit(&sh->free_v[s]);
                mma_commit(&sh->pv_done);
                if (j == n_tiles - 1) mma_commit(&sh->all_done);  // once, after the last P.V
                if (j + 2 < n_tiles && !issue_qk(j + 2)) { ngive_up(sh, 33); break; }  // over the P tile P.V(j) has just read
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
            if (!__all_sync(0xffffffffu, nwait(&sh->q_full, 0, sh))) ngive_up(sh, 39), ok = false;
            if (p.rope && t < p.T) rotate_q(sV, tid, p.rope + (long long)t * (p.dim_out >> 1), p.dim_out >> 3, 0, p.dim_out >> 3);
            float4 x[D / 4];
#pragma unroll
            for (int c = 0; c < D / 4; ++c) x[c] = *q_at(sV, tid, c), top = fmaxf(top, max_abs4(x[c]));
            const float mq = block_mult(__float_as_uint(top));
#pragma unroll
            for (int cb = 0; cb < D / 32; ++cb) {
                uint32_t qh[16], ql[16];
                split_q32([&](int c) { return x[cb * 8 + c]; }, mq, qh, ql);
                tmem_st16(tmem + lane_base + cQh + cb * 16, qh);
                tmem_st16(tmem + lane_base + cQl + cb * 16, ql);
            }
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive_warp(&sh->a_ready);
        }
        pdl_wait();
        const float mk = block_mult(p.amax_k[b * p.n_kv_heads + g]), mv = block_mult(p.amax_v[b * p.n_kv_heads + g]);
        publish_q_top(p, b * p.n_kv_heads + g, top);
        const float cs = score_scale(p.scale_log2, block_mult(__float_as_uint(top)), mk);
        float m_ref = -INFINITY, l = 0.f;
        float m_flushed = -INFINITY;  // the reference maximum of what has been flushed
        const long long row_at = (((long long)b * p.T + t) * p.n_heads + h) * p.dim_out;
        const FlushRow row{FLUSH && t < p.T ? p.out + row_at : nullptr, p.dim_out};
        for (int j = 0; ok && j < n_tiles; ++j) {
            if (!__all_sync(0xffffffffu, nwait(&sh->s_full[j & 1], (uint32_t)((j >> 1) & 1), sh))) {
                ngive_up(sh, 35);
                ok = false;
                break;
            }
            tc_fence_after();
            const int s0 = j * BN;
            const uint32_t sp = tmem + lane_base + cS0 + (j & 1) * BN;
            const bool diag = (s0 + BN - 1 > p.q_offset + t0 + warp * 32) && !ZT_DEFECT(1);
            uint32_t r0[32], r1[32];
            tmem_ld32(sp, r0);
            tmem_ld32(sp + 32, r1);
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
                if (!__all_sync(0xffffffffu, nwait(&sh->pv_done, (uint32_t)((j - 1) & 1), sh))) {
                    ngive_up(sh, 36);
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
                        tmem_ld32(tmem + lane_base + cO + c, r);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * factor);
                        tmem_st32(tmem + lane_base + cO + c, r);
                    }
                }
            }
            // l is kept in P's units (times kPScale), like O
            const float off = ((m_ref == -INFINITY) ? 0.f : m_ref) - 7.0f;  // log2 kPScale
            uint32_t ph[16], pl[16];
            float psum = row_exp32(r0, cs, off, ph, pl);
            tmem_st16(sp, ph);
            tmem_st16(sp + 16, pl);
            psum += row_exp32(r1, cs, off, ph, pl);
            tmem_st16(sp + 32, ph);
            tmem_st16(sp + 48, pl);
            l += psum;
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive_warp(&sh->p_full[j & 1]);
        }
        if (ok && !__all_sync(0xffffffffu, nwait(&sh->all_done, 0, sh))) {
            ngive_up(sh, 38);
            ok = false;
        }
        // the rows go to global memory through K's slots, as in attn_fwd_tc16
        constexpr int RS = D * 4 + 16;
        const bool plain = p.o_planes == nullptr && p.out_peers.n == 0;
        uint8_t *srow = sK + tid * RS;
        if (ok) {
            tc_fence_after();
            const float inv = 1.f / (l * mv);  // l, like O, carries kPScale
            const bool add = FLUSH && m_flushed != -INFINITY && row.sums != nullptr;
            const float ff = add ? ex2(m_flushed - m_ref) : 0.f;
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                uint32_t ra[32];
                tmem_ld32(tmem + lane_base + cO + c, ra);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    float4 o4 = make_float4(__uint_as_float(ra[i]), __uint_as_float(ra[i + 1]), __uint_as_float(ra[i + 2]), __uint_as_float(ra[i + 3]));
                    if (add && c + i < row.width) o4 = flush_sum4(row.sums + c + i, ff, false, o4);
                    o4.x *= inv, o4.y *= inv, o4.z *= inv, o4.w *= inv;
                    *reinterpret_cast<float4 *>(srow + (c + i) * 4) = o4;
                }
            }
            if (p.lse && t < p.T) p.lse[((long long)b * p.T + t) * p.n_heads + h] = (m_ref + log2f(l) - 7.0f) * kLn2;
        }
        if (plain) send_row<FLUSH>(p.out + row_at, srow, p.dim_out, ok && t < p.T);
        mbar_arrive_warp(&sh->staged);
        if (!plain && __all_sync(0xffffffffu, nwait(&sh->staged, 0, sh)) && !sh->abort) {
            const long long wo = (long long)p.n_heads * p.dim_out;
            const float mo = p.o_planes ? out_plane_mult(p, b) : 1.f;
            const int ch = lane & 15;
#pragma unroll 4
            for (int i = 0; i < 32; i += 2) {  // two rows an instruction
                const int r = warp * 32 + i + (lane >> 4);
                const float4 o4 = *reinterpret_cast<const float4 *>(sK + r * RS + ch * 16);
                if (t0 + r < p.T && ch * 4 < p.dim_out)  // (a padded tile's upper columns are not the tensor's)
                    store_out4(p, ((long long)b * p.T + t0 + r) * wo + (long long)h * p.dim_out + ch * 4, o4, mo);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 5) tmem_dealloc(tmem, 256);
}

inline int launch_n(const CUtensorMap &kmap, const CUtensorMap &vmap, const CUtensorMap &qmap, Params p, int sms, cudaStream_t stream) {
    const size_t smem = 12 * (size_t)(64 * 64 * 2) + sizeof(SharedN);
    const auto kernel = with_flags([](auto flush, auto pad) { return attn_fwd_tc16n<flush.value, pad.value>; }, p.flush, head_steps(p.dim_out) < 4);
    if (optin_smem((const void *)kernel, smem)) return 1;
    const unsigned tiles = (unsigned)((p.T + 127) / 128), heads = (unsigned)p.n_heads, seqs = (unsigned)p.batch;
    // Tile by tile up to four waves, where the tail counts, and to eight where the planes of k and v of all sequences stay in L2 (two halves of
    // 63 MB), else sequence by sequence.  Us by tile / by sequence: 16/16 heads, 2 of T 3000 (768 blocks) 93 / 110; 12/4, 4 of 2000
    // (768) 70 / 81; 32/8, 8 of 1024 (2048 blocks, 34 MB) 110 / 124; 16/16 of 32 columns, 4 of 4096 (2048, 67 MB) 376 / 340; 32/8, 64 of
    // 140 (4096) 144 / 129, 16 of 1024 (4096) 283 / 255, 8 of 4096 (8192) 1449 / 1397; few long ones lose a little, 2 of 8000 1308 / 1357.
    const long long blocks = (long long)tiles * heads * seqs, kv = 8LL * p.batch * (p.q_offset + p.T) * p.n_kv_heads * plane_dim(p.dim_out);
    p.by_tile = blocks <= 8LL * sms || (blocks <= 16LL * sms && kv <= (48LL << 20));
    return launch_after("attn_fwd_tc16n", kernel, p.by_tile ? dim3(heads * seqs * tiles) : dim3(tiles, heads, seqs), dim3(kThreadsN), smem, stream, 2, kmap, vmap, qmap, p);
}

}  // namespace tcf16
}  // namespace zt
