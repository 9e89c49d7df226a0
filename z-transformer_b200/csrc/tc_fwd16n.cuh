// attn_fwd_tc16n: the f16-split forward of heads of up to 64 columns (narrower ones padded), two CTAs an SM.
//
// A tile of 64 keys is 768 clocks of MMAs here, half of what it is at 128 columns, while its softmax is as long as there: with one CTA
// an SM, two heads in it (attn_fwd_tc16g), a pair of tiles took 2700 clocks where the MMAs take 1660, and on the way to the first MMA
// and from the last one to memory (12000 clocks) nothing at all ran.  Two CTAs fill each other's gaps.  What makes room for the
// second:
//   CTA    128 query rows of ONE head; 6 warps: four softmax warps (a thread per row, every key tile), TMA, MMA.
//   TMEM   [0, 128) two accumulators of O, [128, 256) two S/P tiles of 64 columns: half of it.
//   smem   the query tile (f32, then its hi and lo pieces: S is made of SS MMAs, 960 clocks a key tile in all), K ring of three slots, V ring of
//          two: 112 KB.  The rows leave through K's slots.
//   MMA    S(0) S(1) | P.V(0) S(2) | P.V(1) S(3) | ...: the softmax of tile j+1 runs under P.V(j) and S(j+2).
// The arithmetic is attn_fwd_tc16's, bit for bit: key tiles of either parity have an accumulator, a reference maximum and a sum of their own, which
// halves what O loses to truncation.  (With Q in tensor memory and one accumulator a launch took a tenth less, and out's error against float64 rose
// by half and more: T 512, 16/16 heads 6.2e-7 -> 8.6e-7, T 2000 1.25e-6 -> 2.2e-6.)
// Us of the kernel, the forms before (one or two heads a CTA, whichever took the call) -> this: batch 8, T 512, 32/8 heads 64 -> 53; 2 of T
// 3000, 16/16 heads 146 -> 103; 4 of 2000, 12/4 113 -> 76; 8 of 700, 12/4 54 -> 35; 64 of 256, 12/4 100 -> 72; 16 of 130, 16/16 of 32
// columns 35 -> 21.  (Two heads a CTA, one CTA an SM, with two S buffers each and the next
// tiles' rows split ahead: 64 -> 54, 146 -> 121, 113 -> 87.)
#pragma once

#include "tc_fwd16.cuh"

namespace zt {
namespace tcf16 {

constexpr int kThreadsN = 6 * 32;

struct SharedN {
    uint64_t full_k[3], free_k[3], full_v[2], free_v[2];
    uint64_t a_ready, q_full, s_full[2], p_full[2], staged, all_done;
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
    constexpr int cO0 = 0, cS0 = 128;  // O of the tiles of parity s at cO0 + 64 s, S/P at cS0 + 64 s
    const bool padded = PAD && plane_dim(p.dim_out) < D;  // the planes are narrower than the tile
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *sK = smem_raw, *sV = sK + 6 * KP, *sQ = sV + 4 * KP;
    SharedN *sh = reinterpret_cast<SharedN *>(sQ + 4 * KP);

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
        for (int i = 0; i < 3; ++i) mbar_init(&sh->full_k[i], 1), mbar_init(&sh->free_k[i], 1);
        mbar_init(&sh->a_ready, 4), mbar_init(&sh->q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh->full_v[i], 1), mbar_init(&sh->free_v[i], 1);
            mbar_init(&sh->s_full[i], 1), mbar_init(&sh->p_full[i], 4);
        }
        mbar_init(&sh->staged, 4), mbar_init(&sh->all_done, 1);
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
            load_q<D>(sQ, &qmap, &sh->q_full, t0, h, b);
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
                const int s = j & 1;
                if (j >= 2 && !nwait(&sh->free_v[s], (uint32_t)(((j >> 1) & 1) ^ 1), sh)) { ngive_up(sh, 31), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_v[s], 2 * KP);
                load_head<1>(sV + s * 2 * KP, &vmap, &sh->full_v[s], j * BN, g, b, BN * 128, padded);
                load_head<1>(sV + s * 2 * KP + KP, &vmap, &sh->full_v[s], j * BN, g, B + b, BN * 128, padded);
                ++n_v;
            };
            load_k(0);
            if (n_tiles > 1) load_k(1);
            for (int j = 0; live && j < n_tiles; ++j) {  // (S runs two key tiles ahead of P.V)
                load_v(j);
                if (live && j + 2 < n_tiles) load_k(j + 2);
            }
            if (sh->abort) {
                // let the copies in flight land before the CTA's shared memory goes away
                mbar_wait(&sh->q_full, 0);
                for (int j = (n_k > 3 ? n_k - 3 : 0); j < n_k; ++j) mbar_wait(&sh->full_k[j % 3], (uint32_t)((j / 3) & 1));
                for (int j = (n_v > 2 ? n_v - 2 : 0); j < n_v; ++j) mbar_wait(&sh->full_v[j & 1], (uint32_t)((j >> 1) & 1));
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
            const uint64_t bqh = desc_kmajor(smem_u32(sQ)), bql = desc_kmajor(smem_u32(sQ) + kQBlock);
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
                    mma_ss_f16(tmem + cS, desc_advance(bqh, kk * 32), dkh, id_s, kk > 0);
                    mma_ss_f16(tmem + cS, desc_advance(bqh, kk * 32), dkl, id_s, 1);
                    mma_ss_f16(tmem + cS, desc_advance(bql, kk * 32), dkh, id_s, 1);
                }
                mma_commit(&sh->free_k[s]);
                mma_commit(&sh->s_full[j & 1]);
                return true;
            };
            if (ok && !issue_qk(0)) { ngive_up(sh, 33); ok = false; }
            if (ok && n_tiles > 1 && !issue_qk(1)) { ngive_up(sh, 33); ok = false; }
            for (int j = 0; ok && j < n_tiles; ++j) {
                const int s = j & 1;
                if (!nwait(&sh->p_full[s], (uint32_t)((j >> 1) & 1), sh) ||
                    !nwait(&sh->full_v[s], (uint32_t)((j >> 1) & 1), sh)) { ngive_up(sh, 34); break; }
                tc_fence_after();
                const bool fresh = j < 2 || (FLUSH && (j >> 1) % kFlushKeyTiles == 0);  // (O was flushed before tile j)
                const uint32_t vh = v_u32 + (uint32_t)(s * 2 * KP);
                const uint64_t mvh = desc_mnmajor_16b(vh, BN * 128), mvl = desc_mnmajor_16b(vh + KP, BN * 128);
                const uint32_t cS = cS0 + s * BN, cO = cO0 + s * D;
#pragma unroll
                for (int kk = 0; kk < BN / 16; ++kk) {
                    const uint32_t ac = (uint32_t)(32 * (kk >> 1) + (kk & 1) * 8);
                    const uint64_t dvh = desc_advance(mvh, kk * 2048), dvl = desc_advance(mvl, kk * 2048);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvh, id_o, (!fresh || kk > 0) ? 1 : 0);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvl, id_o, 1);
                    mma_ts_f16(tmem + cO, tmem + cS + ac + 16, dvh, id_o, 1);
                }
                mma_commit(&sh->free_v[s]);
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
            if (p.rope && t < p.T) rotate_q(sQ, tid, p.rope + (long long)t * (p.dim_out >> 1), p.dim_out >> 3, 0, p.dim_out >> 3);
            float4 x[D / 4];
#pragma unroll
            for (int c = 0; c < D / 4; ++c) x[c] = *q_at(sQ, tid, c), top = fmaxf(top, max_abs4(x[c]));
            const float mq = block_mult(__float_as_uint(top));
#pragma unroll
            for (int cb = 0; cb < D / 32; ++cb) {
                uint32_t qh[16], ql[16];
                split_q32([&](int c) { return x[cb * 8 + c]; }, mq, qh, ql);
                store_q_piece(sQ, tid, cb, qh), store_q_piece(sQ + kQBlock, tid, cb, ql);  // (over the row's own f32)
            }
            fence_async_smem();
            mbar_arrive_warp(&sh->a_ready);
        }
        pdl_wait();
        const float mk = block_mult(p.amax_k[b * p.n_kv_heads + g]), mv = block_mult(p.amax_v[b * p.n_kv_heads + g]);
        publish_q_top(p, b * p.n_kv_heads + g, top);
        const float cs = score_scale(p.scale_log2, block_mult(__float_as_uint(top)), mk);
        // of the tiles of either parity: the reference maximum, the sum, the reference maximum of what has been flushed, and where that is kept
        float m_of[2] = {-INFINITY, -INFINITY}, l_of[2] = {0.f, 0.f}, f_of[2] = {-INFINITY, -INFINITY};
        const long long row_at = (((long long)b * p.T + t) * p.n_heads + h) * p.dim_out;
        FlushRow row0{}, row1{};
        if (FLUSH) row0 = flush_row_at(p, p.out, b, t0 + warp * 32, h), row1 = flush_row_at(p, p.flush_rows, b, t0 + warp * 32, h);
        const auto softmax = [&](int j, auto parity) -> bool {
            constexpr int s = parity.value;
            float &m_ref = m_of[s], &l = l_of[s], &m_flushed = f_of[s];
            if (!__all_sync(0xffffffffu, nwait(&sh->s_full[s], (uint32_t)((j >> 1) & 1), sh))) {
                ngive_up(sh, 35);
                return false;
            }
            tc_fence_after();
            const int s0 = j * BN;
            const uint32_t sp = tmem + lane_base + cS0 + s * BN, cO = cO0 + s * D;
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
            const bool flush = FLUSH && j > 1 && (j >> 1) % kFlushKeyTiles == 0;
            const bool moved = __any_sync(0xffffffffu, factor != 1.f);
            if (j > 1 && (flush || moved)) {  // (the accumulator's last P.V, j - 2, retired before S(j), which was issued behind it)
                if (flush) {
                    const bool first = m_flushed == -INFINITY;
                    flush_row<D>(tmem + lane_base + cO, s == 0 ? row0 : row1, first ? 0.f : ex2(m_flushed - m_old), first);
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
            mbar_arrive_warp(&sh->p_full[s]);
            return true;
        };
        for (int j = 0; ok && j < n_tiles; j += 2) {
            ok = softmax(j, std::integral_constant<int, 0>{});
            if (ok && j + 1 < n_tiles) ok = softmax(j + 1, std::integral_constant<int, 1>{});
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
            const bool two = n_tiles > 1;  // the odd accumulator holds something only then
            const float m0 = m_of[0], m1 = two ? m_of[1] : -INFINITY, l0 = l_of[0], l1 = two ? l_of[1] : 0.f;
            const float mm = fmaxf(fmaxf(m0, m1), -3.0e38f);
            // (the merge is a running-maximum correction too, the only one where each parity has a single tile)
            const float w0 = ZT_DEFECT(3) ? 1.f : ex2(m0 - mm), w1 = (m1 == -INFINITY) ? 0.f : (ZT_DEFECT(3) ? 1.f : ex2(m1 - mm));
            const float lsum = w0 * l0 + w1 * l1;
            const float inv = lsum == 0.f ? 0.f : 1.f / (lsum * mv);  // lsum, like O, carries kPScale
            const float f0 = w0 * inv, f1 = w1 * inv;
            const bool add0 = FLUSH && f_of[0] != -INFINITY && row0.sums != nullptr, add1 = FLUSH && f_of[1] != -INFINITY && row1.sums != nullptr;
            const float g0 = add0 ? ex2(f_of[0] - m0) : 0.f, g1 = add1 ? ex2(f_of[1] - m1) : 0.f;
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                uint32_t ra[32], rb[32];
                tmem_ld32(tmem + lane_base + cO0 + c, ra);
                if (two) tmem_ld32(tmem + lane_base + cO0 + D + c, rb);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    float4 o4 = make_float4(__uint_as_float(ra[i]), __uint_as_float(ra[i + 1]), __uint_as_float(ra[i + 2]), __uint_as_float(ra[i + 3]));
                    if (add0 && c + i < row0.width) o4 = flush_sum4(row0.at(c + i), g0, false, o4);
                    o4.x *= f0, o4.y *= f0, o4.z *= f0, o4.w *= f0;
                    if (two && w1 != 0.f) {
                        float4 x4 = make_float4(__uint_as_float(rb[i]), __uint_as_float(rb[i + 1]), __uint_as_float(rb[i + 2]), __uint_as_float(rb[i + 3]));
                        if (add1 && c + i < row1.width) x4 = flush_sum4(row1.at(c + i), g1, false, x4);
                        o4.x += x4.x * f1, o4.y += x4.y * f1, o4.z += x4.z * f1, o4.w += x4.w * f1;
                    }
                    *reinterpret_cast<float4 *>(srow + (c + i) * 4) = o4;
                }
            }
            if (p.lse && t < p.T) p.lse[((long long)b * p.T + t) * p.n_heads + h] = (mm + log2f(lsum) - 7.0f) * kLn2;
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
    const size_t smem = 14 * (size_t)(64 * 64 * 2) + sizeof(SharedN);
    const auto kernel = with_flags([](auto flush, auto pad) { return attn_fwd_tc16n<flush.value, pad.value>; }, p.flush, head_steps(p.dim_out) < 4);
    if (optin_smem((const void *)kernel, smem)) return 1;
    const unsigned tiles = (unsigned)((p.T + 127) / 128), heads = (unsigned)p.n_heads, seqs = (unsigned)p.batch;
    // Tile by tile up to eight blocks an SM, where the tail counts, and beyond where the planes of k and v of all sequences stay in L2 (two
    // halves of 63 MB), else sequence by sequence.  Us a forward, back to back for most of a second, by tile / by sequence: 16/16 heads, 2 of T
    // 3000 (5 blocks an SM) 130 / 162; 12/4, 4 of 2000 (5) 89 / 108; 64 MB of planes: 32/8, 2 of 8192 (28) 1513 / 1567, 12/4, 16 of 2048 (21)
    // 383 / 386, 32/8 of 32 columns, 100 of 300 (65) 356 / 382; 128 MB: 32/8, 8 of 4096 (55) 1742 / 1688, 16/4, 32 of 2048 (55) 1014 /
    // 976, 16/16, 8 of 2048 (14) 329 / 319, 2 of 8000 (14) 841 / 867, 32/8, 64 of 512 (55) 456 / 468, one of 32768 11124 / 11117; 256 MB:
    // 16/16 of 32 columns, 16 of 4096 (55) 1606 / 1431.
    const long long blocks = (long long)tiles * heads * seqs, kv = 8LL * p.batch * (p.q_offset + p.T) * p.n_kv_heads * plane_dim(p.dim_out);
    p.by_tile = blocks <= 8LL * sms || kv <= (64LL << 20);
    return launch_after("attn_fwd_tc16n", kernel, p.by_tile ? dim3(heads * seqs * tiles) : dim3(tiles, heads, seqs), dim3(kThreadsN), smem, stream, 2, kmap, vmap, qmap, p);
}

}  // namespace tcf16
}  // namespace zt
