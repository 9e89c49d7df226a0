// attn_fwd_tc16 for two query heads of one KV group per CTA.
//
// The forward moves 64 KB of K and V (hi and lo planes) from L2 into an SM per 64-key tile and 128 query
// rows, 7 TB/s over the whole chip at the headline shape, and that traffic bounds it as much as its MMAs do.
// The heads of a KV group read the same K and V: here a CTA takes the same 128 query rows of two of them and
// uses every K/V tile it loads twice, which halves the traffic.  The two softmax warp sets, which in
// attn_fwd_tc16 split one head's key tiles between them by parity, take one head each and walk every tile:
//   TMEM  [0, D/2) Qh of head A, [D/2, D) Qh of head B, [D, 2D) O of A, [2D, 3D) O of B, then S/P of A and of B
//         (64 columns each): the Q lo planes, needed by one of the three split terms, stay in shared memory
//         (an SS MMA), which is what makes room for the second head;
//   MMA   S_A(0) S_B(0) | P.V_A(j) S_A(j+1) P.V_B(j) S_B(j+1) | ...: a head's next S goes out behind its P.V,
//         so its softmax runs under the other head's MMAs, as with the parity split;
//   smem  K ring of three slots, V ring of two, the lo pieces of two query tiles (224 KB at head_dim 128).
// One accumulator per head: no merge at the end.  Needs an even number of query heads per KV group.
#pragma once

#include "tc_fwd16.cuh"

namespace zt {
namespace tcf16 {

struct SharedG {
    uint64_t full_k[3], free_k[3], full_v[2], free_v[2];
    uint64_t a_ready[2], q_full[2], s_full[2], p_full[2], pv_done[2], staged[2], all_done;
    uint32_t tmem_base;
    volatile int abort;
    float q_top[2][2][128];  // of a head: max |q| of each half of a row's columns
};
__device__ __forceinline__ bool gwait(uint64_t *bar, uint32_t parity, SharedG *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}
__device__ __forceinline__ void ggive_up(SharedG *sh, int code) {
    sh->abort = code;
    atomicMax(&g_tc_status, code);
}

template <int D, bool FLUSH, bool PAD>
__global__ void __launch_bounds__(kThreads, 1)
    attn_fwd_tc16g(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                   const __grid_constant__ CUtensorMap qmap, const Params p) {
    constexpr int NB = D / 64, W2 = D / 2, BN = 64;
    constexpr int KP = BN * D * 2;  // bytes of one plane of a key tile; a ring slot is 2 KP (hi, lo)
    const bool padded = PAD && plane_dim(p.dim_out) < D;  // the planes are narrower than the tile
    constexpr int cQh = 0, cO0 = D, cS0 = 3 * D;  // head s: Qh at cQh + s W2, O at cO0 + s D, S/P at cS0 + 64 s
    extern __shared__ __align__(1024) uint8_t smem_raw[];  // (the swizzled tiles need the alignment; checked below)
    // Behind K's ring: head s's f32 query tile at sQ + s 4 KP, of which its lo pieces take the first half over and V's slot s the other.
    uint8_t *sK = smem_raw, *sQ = sK + 6 * KP;
    SharedG *sh = reinterpret_cast<SharedG *>(sQ + 8 * KP);

    const int warp = threadIdx.x >> 5;
    // launch order (x fastest): the head pairs of a sequence, query tile by query tile, late (long) tiles first, so
    // that the last CTAs to start are the shortest (1.5 % faster than a head pair's tiles together)
    const int qt = (int)gridDim.y - 1 - (int)blockIdx.y;
    // (the sequences are along z, or along x behind each other: see tile_by_tile)
    const int pairs = p.n_heads / 2, bx = (int)blockIdx.x / pairs, h0 = 2 * ((int)blockIdx.x - bx * pairs), b = (int)blockIdx.z + bx;
    const int g = h0 / (p.n_heads / p.n_kv_heads);
    const int t0 = qt * 128;
    const int rows_end = (t0 + 128 < p.T) ? t0 + 128 : p.T;
    const int n_tiles = (p.q_offset + rows_end + BN - 1) / BN;
    const int B = p.batch;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 3; ++i) mbar_init(&sh->full_k[i], 1), mbar_init(&sh->free_k[i], 1);
        for (int i = 0; i < 2; ++i) mbar_init(&sh->full_v[i], 1), mbar_init(&sh->free_v[i], 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh->s_full[i], 1), mbar_init(&sh->p_full[i], 4), mbar_init(&sh->pv_done[i], 1);
            mbar_init(&sh->staged[i], 4);
            mbar_init(&sh->q_full[i], 1), mbar_init(&sh->a_ready[i], 8);
        }
        mbar_init(&sh->all_done, 1);
        sh->abort = (smem_u32(smem_raw) & 1023u) ? 40 : 0;
        if (sh->abort) atomicMax(&g_tc_status, 40);
        mbar_fence_init();
    }
    if (warp == 9) tmem_alloc(&sh->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    // (the query rows are older than the launch before this one, for whose planes and maxima pdl_wait() waits)

    if (warp == 8) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one() && !sh->abort) {
            tma_prefetch_desc(&qmap), tma_prefetch_desc(&kmap), tma_prefetch_desc(&vmap);
            for (int i = 0; i < 2; ++i) {
                mbar_arrive_expect_tx(&sh->q_full[i], 4 * KP);
                load_q<D>(sQ + i * 4 * KP, &qmap, &sh->q_full[i], t0, h0 + i, b);
            }
            pdl_wait();
            pdl_launch();
            int n_k = 0, n_v = 0;  // tiles issued
            bool live = true;
            auto load_k = [&](int j) {
                const int s = j % 3;
                if (j >= 3 && !gwait(&sh->free_k[s], (uint32_t)(((j / 3) & 1) ^ 1), sh)) { ggive_up(sh, 41), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_k[s], 2 * KP);
                load_head<NB>(sK + s * 2 * KP, &kmap, &sh->full_k[s], j * BN, g, b, BN * 128, padded);
                load_head<NB>(sK + s * 2 * KP + KP, &kmap, &sh->full_k[s], j * BN, g, B + b, BN * 128, padded);
                ++n_k;
            };
            auto load_v = [&](int j) {
                const int s = j & 1;
                if (j >= 2 && !gwait(&sh->free_v[s], (uint32_t)(((j >> 1) & 1) ^ 1), sh)) { ggive_up(sh, 41), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_v[s], 2 * KP);
                load_head<NB>(sQ + (2 + 4 * s) * KP, &vmap, &sh->full_v[s], j * BN, g, b, BN * 128, padded);
                load_head<NB>(sQ + (3 + 4 * s) * KP, &vmap, &sh->full_v[s], j * BN, g, B + b, BN * 128, padded);
                ++n_v;
            };
            for (int j = 0; j < 3 && j < n_tiles; ++j) load_k(j);
            for (int j = 0; live && j < 2 && j < n_tiles; ++j) {
                if (!gwait(&sh->a_ready[j], 0, sh)) ggive_up(sh, 41), live = false;
                else load_v(j);
            }
            for (int j = 2; live && j < n_tiles; ++j) {
                if (j + 1 < n_tiles) load_k(j + 1);
                if (live) load_v(j);
            }
            if (sh->abort) {
                // let the copies in flight land before the CTA's shared memory goes away
                mbar_wait(&sh->q_full[0], 0), mbar_wait(&sh->q_full[1], 0);
                for (int j = (n_k > 3 ? n_k - 3 : 0); j < n_k; ++j) mbar_wait(&sh->full_k[j % 3], (uint32_t)((j / 3) & 1));
                for (int j = (n_v > 2 ? n_v - 2 : 0); j < n_v; ++j) mbar_wait(&sh->full_v[j & 1], (uint32_t)((j >> 1) & 1));
            }
        }
        __syncwarp();
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t id_s = idesc_f16(128, BN, false, false);
            const int steps = PAD ? head_steps(p.dim_out) : D / 16;
            const uint32_t id_o = idesc_f16(128, 16 * steps, false, true);
            bool ok = true;
            const uint32_t k_u32 = smem_u32(sK), q_u32 = smem_u32(sQ);
            // S of head `hd`, tile j (K tile j has landed: the caller waited)
            auto issue_qk = [&](int hd, int j) {
                const uint32_t kh = k_u32 + (uint32_t)((j % 3) * 2 * KP);
                const uint64_t bkh = desc_kmajor(kh), bkl = desc_kmajor(kh + KP);
                const uint64_t bql = desc_kmajor(q_u32 + (uint32_t)(hd * 4 * KP));
                const uint32_t cS = cS0 + hd * BN, cQ = cQh + hd * W2;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    if (PAD && kk >= steps) break;
                    const uint32_t ao = (uint32_t)((kk >> 2) * (128 * 128) + (kk & 3) * 32);
                    const uint32_t bo = (uint32_t)((kk >> 2) * (BN * 128) + (kk & 3) * 32);
                    const uint64_t dkh = desc_advance(bkh, bo), dkl = desc_advance(bkl, bo);
                    mma_ts_f16(tmem + cS, tmem + cQ + kk * 8, dkh, id_s, kk > 0);
                    mma_ts_f16(tmem + cS, tmem + cQ + kk * 8, dkl, id_s, 1);
                    mma_ss_f16(tmem + cS, desc_advance(bql, ao), dkh, id_s, 1);
                }
                if (hd == 1) mma_commit(&sh->free_k[j % 3]);
                mma_commit(&sh->s_full[hd]);
            };
            auto k_landed = [&](int j) -> bool {
                if (!gwait(&sh->full_k[j % 3], (uint32_t)((j / 3) & 1), sh)) return false;
                tc_fence_after();
                return true;
            };
            // P.V of head `hd`, tile j (V tile j has landed)
            auto issue_pv = [&](int hd, int j) {
                const bool fresh = j == 0 || (FLUSH && j % kFlushKeyTiles == 0);  // (O was flushed before tile j)
                const uint32_t vh = q_u32 + (uint32_t)((2 + 4 * (j & 1)) * KP);
                const uint64_t mvh = desc_mnmajor_16b(vh, BN * 128), mvl = desc_mnmajor_16b(vh + KP, BN * 128);
                const uint32_t cS = cS0 + hd * BN, cO = cO0 + hd * D;
#pragma unroll
                for (int kk = 0; kk < BN / 16; ++kk) {
                    const uint32_t ac = (uint32_t)(32 * (kk >> 1) + (kk & 1) * 8);
                    const uint64_t dvh = desc_advance(mvh, kk * 2048), dvl = desc_advance(mvl, kk * 2048);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvh, id_o, (!fresh || kk > 0) ? 1 : 0);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvl, id_o, 1);
                    mma_ts_f16(tmem + cO, tmem + cS + ac + 16, dvh, id_o, 1);
                }
                if (hd == 1) mma_commit(&sh->free_v[j & 1]);
                mma_commit(&sh->pv_done[hd]);
            };
            for (int hd = 0; ok && hd < 2; ++hd) {
                if (!gwait(&sh->a_ready[hd], 0, sh) || !k_landed(0)) { ggive_up(sh, 42); ok = false; }
                else issue_qk(hd, 0);
            }
            for (int j = 0; ok && j < n_tiles; ++j) {
                const uint32_t par = (uint32_t)(j & 1);
                if (!gwait(&sh->p_full[0], par, sh) || !gwait(&sh->full_v[j & 1], (uint32_t)((j >> 1) & 1), sh)) { ggive_up(sh, 44); break; }
                tc_fence_after();
                issue_pv(0, j);
                if (j + 1 < n_tiles) {
                    if (!k_landed(j + 1)) { ggive_up(sh, 43); break; }
                    issue_qk(0, j + 1);  // overwrites the P tile that P.V_A(j) has just read
                }
                if (!gwait(&sh->p_full[1], par, sh)) { ggive_up(sh, 44); break; }
                tc_fence_after();
                issue_pv(1, j);
                if (j == n_tiles - 1) mma_commit(&sh->all_done);  // once, after the last P.V
                if (j + 1 < n_tiles) issue_qk(1, j + 1);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ softmax rows: set `set` owns
        // head h0 + set, every key tile of it
        const int tid = threadIdx.x & 127, set = threadIdx.x >> 7;
        const int lane = threadIdx.x & 31;
        const int h = h0 + set;
        const int t = t0 + tid, pos = p.q_offset + t;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        bool ok = true;
        float top = 0.f;  // max |q| of the row
        {
            // both sets take one head's rows, then the other's: the first head's S runs under the second's conversion
            const float2 *angles = p.rope ? p.rope + (long long)(t < p.T ? t : 0) * (p.dim_out >> 1) : nullptr;
#pragma unroll
            for (int hd = 0; hd < 2; ++hd) {
                if (!__all_sync(0xffffffffu, gwait(&sh->q_full[hd], 0, sh))) ggive_up(sh, 49), ok = false;
                const float x = convert_q<D, true>(sQ + hd * 4 * KP, set, tid, angles, p.dim_out, sh->q_top[hd], tmem + lane_base + cQh + hd * W2, 0u);
                if (hd == set) top = x;
                mbar_arrive_warp(&sh->a_ready[hd]);
            }
        }
        pdl_wait();
        const float mk = block_mult(p.amax_k[b * p.n_kv_heads + g]), mv = block_mult(p.amax_v[b * p.n_kv_heads + g]);
        publish_q_top(p, b * p.n_kv_heads + g, top);
        const float cs = score_scale(p.scale_log2, block_mult(__float_as_uint(top)), mk);
        const uint32_t cS = cS0 + set * BN, cO = cO0 + set * D;
        float m_ref = -INFINITY, l = 0.f;
        float m_flushed = -INFINITY;  // the reference maximum of what has been flushed
        FlushRow row{};
        if (FLUSH) row = flush_row_at(p, p.out, b, t0 + (warp & 3) * 32, h);
        for (int j = 0; ok && j < n_tiles; ++j) {
            if (!__all_sync(0xffffffffu, gwait(&sh->s_full[set], (uint32_t)(j & 1), sh))) {
                ggive_up(sh, 45);
                ok = false;
                break;
            }
            tc_fence_after();
            const int s0 = j * BN;
            const bool diag = (s0 + BN - 1 > p.q_offset + t0 + (warp & 3) * 32) && !ZT_DEFECT(1);
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
                // this head's O may only be touched once its previous P.V has retired
                if (!__all_sync(0xffffffffu, gwait(&sh->pv_done[set], (uint32_t)((j - 1) & 1), sh))) {
                    ggive_up(sh, 46);
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
            mbar_arrive_warp(&sh->p_full[set]);
        }
        if (ok && !__all_sync(0xffffffffu, gwait(&sh->all_done, 0, sh))) {
            ggive_up(sh, 48);
            ok = false;
        }
        // The head's rows go to global memory through shared memory (the rings are idle once all_done completes), as in
        // attn_fwd_tc16: 6400 clocks of a CTA by stores of whole rows.
        constexpr int RS = D * 4 + 16;
        const bool plain = p.o_planes == nullptr && p.out_peers.n == 0;
        uint8_t *stage = smem_raw + set * 128 * RS, *srow = stage + tid * RS;
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
                    if (add && c + i < row.width) o4 = flush_sum4(row.at(c + i), ff, false, o4);
                    o4.x *= inv, o4.y *= inv, o4.z *= inv, o4.w *= inv;
                    *reinterpret_cast<float4 *>(srow + (c + i) * 4) = o4;
                }
            }
            if (p.lse && t < p.T) p.lse[((long long)b * p.T + t) * p.n_heads + h] = (m_ref + log2f(l) - 7.0f) * kLn2;
        }
        if (plain) send_row<FLUSH>(p.out + (((long long)b * p.T + t) * p.n_heads + h) * p.dim_out, srow, p.dim_out, ok && t < p.T);
        mbar_arrive_warp(&sh->staged[set]);
        if (!plain && __all_sync(0xffffffffu, gwait(&sh->staged[set], 0, sh)) && !sh->abort) {
            constexpr int CH = D / 4;  // 16-byte chunks per row
            constexpr int RPI = 32 / CH;  // rows per store instruction
            const int ch = lane & (CH - 1);
            const long long wo = (long long)p.n_heads * p.dim_out;
            const float mo = p.o_planes ? out_plane_mult(p, b) : 1.f;
#pragma unroll 4
            for (int i = 0; i < 32; i += RPI) {
                const int r = (warp & 3) * 32 + i + lane / CH;
                const float4 o4 = *reinterpret_cast<const float4 *>(stage + r * RS + ch * 16);
                if (t0 + r < p.T && ch * 4 < p.dim_out)  // (a padded tile's upper columns are not the tensor's)
                    store_out4(p, ((long long)b * p.T + t0 + r) * wo + (long long)h * p.dim_out + ch * 4, o4, mo);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem, 512);
}

template <int D>
inline int launch_g_d(const CUtensorMap &kmap, const CUtensorMap &vmap, const CUtensorMap &qmap, const Params &p,
                      cudaStream_t stream) {
    size_t smem = 14 * (size_t)(64 * D * 2) + sizeof(SharedG);
    if (smem < 120 * 1024) smem = 120 * 1024;  // one CTA per SM: it allocates all of TMEM
    const auto kernel = with_flags([](auto flush, auto pad) { return attn_fwd_tc16g<D, flush.value, pad.value>; }, p.flush, head_steps(p.dim_out) < D / 16);
    if (optin_smem((const void *)kernel, smem)) return 1;
    const dim3 grid = tile_major_grid(p.n_heads / 2, (p.T + 127) / 128, p.batch, kFwdTileWaves);
    return launch_after("attn_fwd_tc16g", kernel, grid, dim3(kThreads), smem, stream, 1, kmap, vmap, qmap, p);
}

}  // namespace tcf16
}  // namespace zt
