// Causal GQA attention backward above head_dim 128, on tiles of 192 and 256 columns, on the tensor cores.
//
// What it computes: autograd.attentionBackward (src/autograd.zig:636-842) for a batch, as tc_bwd.cuh does:
//     P = exp(S - lse),  dP = dO V^T,  dS = P (dP - delta),  dV = P^T dO,  dK = scale dS^T Q,  dQ = scale dS K
// with the same arithmetic (f32 operands as f16 hi/lo planes times a power of two, three kind::f16 MMAs per
// product, f32 accumulation in TMEM).
//
// Why another form.  The fused kernels of tc_bwd.cuh keep a CTA's K, V, Q, dO tiles and the dK, dV (or dQ)
// accumulators on chip at once.  At head_dim 256 that is two 256-column accumulators -- all 512 TMEM columns
// before S and dP have any -- and four 64 KB operand tiles beside them.  Here the products are separate
// launches and P and dS travel through memory, as f16 hi/lo planes laid out as the next launch's operand:
//   bwd_wide_scores   one CTA per (128 query rows, 128 keys) tile at or below the diagonal of one (sequence,
//                     head): S = Q K^T and dP = dO V^T over the head's 256 columns into two TMEM accumulators,
//                     then P and dS, split, into the scratch planes [T, T] of that head;
//   wide_products     dQ = scale dS K: 128 x 256 output tiles (the whole head), contraction over the keys a query tile sees;
//                     dK = scale sum_h dS^T Q and dV = sum_h P^T dO: contraction over the query rows at or after
//                     the key tile, every head of the KV group adding into the same output.
// Contractions longer than 1024 are cut into pieces that separate CTAs add with red.global.add.f32 (the tensor
// core adds into its accumulator with truncation; see tc_gemm.cuh), so dq, dk, dv are zeroed first.
// The planes of P and dS cost 8 bytes per (query, key) pair written and 12 read -- independent of head_dim,
// which is why this form is for the wide heads only: at 256 columns the products above are 2.5 times the flops
// per byte they are at 128.  A scratch of a few GiB holds the planes of a chunk of heads; chunks run in turn.
//
// The scale of dS.  Every query row has its own, from the bound the fused dQ kernel uses (|dS[t, s]| <=
// 2 |dout[t]| max_s |v[s]|): dQ's contraction runs along a row, so the row's factor leaves with the row.  dK's
// contraction runs ACROSS rows, so there the factor is moved to the other operand: the Q planes it reads are a
// second copy whose row t is divided by (row t's scale / the smallest scale of the KV group), a power of two
// between 1 and 2^12, and the product dS Q has one scale again.
#pragma once

#include "tc_gemm.cuh"

namespace zt {
namespace tcw {

using namespace tc;
using tcb::block_mult;
using tcb::kDsBound;
using tcb::ds_group_scale;
using tcb::ds_row_scale;
using tcb::split_pack;
using tcb::fma2;
using tcb::mul2;
using tcb::max3;
using tcb::floats2;
using tcb::clamp_abs;

constexpr int kStages = 3;
constexpr int kTB = 128 * 64 * 2;  // bytes of one plane of an operand tile
constexpr int kSB = 4 * kTB;       // a stage: A hi, A lo, B hi, B lo
constexpr int kScoreThreads = 10 * 32;  // TMA producer, MMA issuer, eight epilogue warps
constexpr int kResThreads = 18 * 32;    // TMA producer, MMA issuer, sixteen row warps
constexpr int kTriThreads = 6 * 32;     // TMA producer, MMA issuer, four epilogue warps
constexpr int kPiece = 1024;            // contraction depth of one unit of wide_products

struct WideShared {
    uint64_t full[kStages], freed[kStages], all_done, staged;
    uint32_t tmem_base;
    volatile int abort;
};
__device__ __forceinline__ bool wwait(uint64_t *bar, uint32_t parity, WideShared *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}
__device__ __forceinline__ void wgive_up(WideShared *sh, int code) {
    sh->abort = code;
    atomicMax(&g_tc_status, code);
}

struct WideParams {
    const float *lse, *delta, *rnorm;  // [B, T, H]
    const uint32_t *amax_q, *amax_k, *amax_v, *amax_do;  // [B, Hkv] bit patterns of max |x|
    const uint32_t *vnmax, *rnmax;     // [B, Hkv] bit patterns: largest row norm of v, of dout (over the group's heads)
    __half *p_planes, *ds_planes;      // [2][unit_cap][Tp][Tp]: hi planes of the chunk's units, then lo planes
    float *dq, *dk, *dv;
    int batch, T, Tp, n_heads, n_kv_heads;
    int dim_out, td;                   // the tensors' head_dim, the planes' (192 or 256)
    int unit0, unit_cap;               // the chunk: units (b * n_heads + h) from unit0; planes allocated for unit_cap
    int units, pieces;                 // wide_products: units of the chunk, pieces of kPiece along one head's contraction
    bool in_turn;                      // and the order of its units (products_in_turn)
    float scale, scale_log2, p_scale;
};

// ---------------------------------------------------------------------------------------------------
// P and dS of one 128 x 128 tile.  grid (tiles at or below the diagonal, units of the chunk), 320 threads.
// Eight 64-deep steps through a ring of three stages: four for S (Q and K tiles), four for dP (dO and V tiles).
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kScoreThreads, 1)
    bwd_wide_scores(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                    const __grid_constant__ CUtensorMap gmap, const __grid_constant__ CUtensorMap vmap, const WideParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    WideShared *sh = reinterpret_cast<WideShared *>(smem_raw + kStages * kSB);
    const int warp = threadIdx.x >> 5;
    // tile (m, n), n <= m, from the index along the triangle
    const int ti = (int)blockIdx.x;
    int m = (int)((sqrtf(8.f * (float)ti + 1.f) - 1.f) * 0.5f);
    while ((m + 1) * (m + 2) / 2 <= ti) ++m;
    while (m * (m + 1) / 2 > ti) --m;
    const int n = ti - m * (m + 1) / 2;
    const int m0 = m * 128, n0 = n * 128;
    const int u = (int)blockIdx.y, ug = p.unit0 + u;
    const int b = ug / p.n_heads, h = ug % p.n_heads;
    const int group = p.n_heads / p.n_kv_heads, g = h / group;
    const int B = p.batch;
    const int nbk = p.td / 64;       // 64-column blocks of a head: steps per product
    const int n_steps = 2 * nbk;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) mbar_init(&sh->full[i], 1), mbar_init(&sh->freed[i], 1);
        mbar_init(&sh->all_done, 1);
        mbar_init(&sh->staged, 8);
        sh->abort = (smem_u32(smem_raw) & 1023u) ? 80 : 0;
        if (sh->abort) atomicMax(&g_tc_status, 80);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&sh->tmem_base, 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait();
    pdl_launch();

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one() && !sh->abort) {
            tma_prefetch_desc(&qmap), tma_prefetch_desc(&kmap), tma_prefetch_desc(&gmap), tma_prefetch_desc(&vmap);
            int issued = 0;
            for (int s = 0; s < n_steps; ++s) {
                const int st = s % kStages;
                if (s >= kStages && !wwait(&sh->freed[st], (uint32_t)(((s / kStages) & 1) ^ 1), sh)) { wgive_up(sh, 81); break; }
                uint8_t *base = smem_raw + st * kSB;
                mbar_arrive_expect_tx(&sh->full[st], 4 * kTB);
                const bool first = s < nbk;
                const int blk = first ? s : s - nbk;
                const CUtensorMap *am = first ? &qmap : &gmap, *bm = first ? &kmap : &vmap;
                tma_load_4d(base, am, &sh->full[st], 0, m0, h * nbk + blk, b);
                tma_load_4d(base + kTB, am, &sh->full[st], 0, m0, h * nbk + blk, B + b);
                tma_load_4d(base + 2 * kTB, bm, &sh->full[st], 0, n0, g * nbk + blk, b);
                tma_load_4d(base + 3 * kTB, bm, &sh->full[st], 0, n0, g * nbk + blk, B + b);
                ++issued;
            }
            if (sh->abort)  // let the copies in flight land before the CTA's shared memory goes away
                for (int s = (issued > kStages ? issued - kStages : 0); s < issued; ++s)
                    mbar_wait(&sh->full[s % kStages], (uint32_t)((s / kStages) & 1));
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_f16(128, 128, false, false);
            const uint32_t s_u32 = smem_u32(smem_raw);
            bool ok = !sh->abort;
            for (int s = 0; ok && s < n_steps; ++s) {
                const int st = s % kStages;
                if (!wwait(&sh->full[st], (uint32_t)((s / kStages) & 1), sh)) { wgive_up(sh, 82); ok = false; break; }
                tc_fence_after();
                const uint32_t base = s_u32 + (uint32_t)(st * kSB);
                const uint64_t ah = desc_kmajor(base), al = desc_kmajor(base + kTB);
                const uint64_t bh = desc_kmajor(base + 2 * kTB), bl = desc_kmajor(base + 3 * kTB);
                const uint32_t acc = tmem + (s < nbk ? 0u : 128u);
                const bool fresh = (s == 0 || s == nbk);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const uint64_t dah = desc_advance(ah, kk * 32), dal = desc_advance(al, kk * 32);
                    const uint64_t dbh = desc_advance(bh, kk * 32), dbl = desc_advance(bl, kk * 32);
                    mma_ss_f16(acc, dah, dbh, idesc, (fresh && kk == 0) ? 0 : 1);
                    mma_ss_f16(acc, dah, dbl, idesc, 1);
                    mma_ss_f16(acc, dal, dbh, idesc, 1);
                }
                mma_commit(&sh->freed[st]);
            }
            if (ok) mma_commit(&sh->all_done);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ a thread per query row and 64 of the
        // tile's 128 keys: warps 2..5 the first 64, warps 6..9 the others
        const int lane = threadIdx.x & 31;
        const int lane_grp = warp & 3;  // the TMEM lanes a warp may read are those of its index modulo 4
        const int half = (warp - 2) >> 2;
        const int row = lane_grp * 32 + lane;
        const uint32_t lane_base = (uint32_t)(lane_grp * 32) << 16;
        const int t = m0 + row;
        const float mq = block_mult(p.amax_q[b * p.n_kv_heads + g]), mk = block_mult(p.amax_k[b * p.n_kv_heads + g]);
        const float mv = block_mult(p.amax_v[b * p.n_kv_heads + g]), mdo = block_mult(p.amax_do[b * p.n_kv_heads + g]);
        const long long ridx = ((long long)b * p.T + (t < p.T ? t : 0)) * p.n_heads + h;
        float cq = 1.f, rel = 1.f;
        if (t < p.T) ds_row_scale(__ldg(p.rnorm + ridx), p.rnmax[b * p.n_kv_heads + g], p.vnmax[b * p.n_kv_heads + g], cq, rel);
        const float cs = p.scale_log2 / (mq * mk);
        // P leaves times p_scale: the factor rides in the exponent
        const float lse2 = (t < p.T) ? __ldg(p.lse + ridx) * kLog2e - log2f(p.p_scale) : 0.f;
        const float c1 = cq / (mdo * mv * p.p_scale);  // (P carries p_scale; dS must not)
        const float dels = (t < p.T && !ZT_DEFECT(13)) ? __ldg(p.delta + ridx) * cq / p.p_scale : 0.f;
        bool ok = __all_sync(0xffffffffu, wwait(&sh->all_done, 0, sh));
        if (!ok) wgive_up(sh, 83);
        bool saturated = false;
        // the four output tiles (P hi, P lo, dS hi, dS lo: 128 rows x 256 bytes each) are put together in the
        // stages, idle by now: 16-byte chunk c of row r at chunk c ^ (r & 15)
        if (ok) {
            tc_fence_after();
            const bool diag = (m == n) || (m0 + 128 > p.T);  // tiles that need the mask
#pragma unroll 1
            for (int c = 0; c < 64; c += 32) {
                uint32_t rs[32], rd[32];
                tmem_ld32(tmem + lane_base + half * 64 + c, rs);
                tmem_ld32(tmem + lane_base + 128 + half * 64 + c, rd);
                tmem_wait_ld();
                const int key0 = n0 + half * 64 + c;
                uint32_t ph[16], pl[16], dh[16], dl[16];
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float pv[2], dv[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int key = key0 + i + e;
                        const bool vis = !diag || ((key <= t || ZT_DEFECT(11)) && key < p.T && t < p.T);
                        const float pe = vis ? ex2(__uint_as_float(rs[i + e]) * cs - lse2) : 0.f;
                        const float x = vis ? pe * (__uint_as_float(rd[i + e]) * c1 - dels) : 0.f;
                        saturated |= !(fabsf(x) <= kDsBound);
                        pv[e] = pe;
                        dv[e] = fminf(fmaxf(x, -kDsBound), kDsBound);
                    }
                    split_pack(pv[0], pv[1], ph[i >> 1], pl[i >> 1]);
                    split_pack(dv[0], dv[1], dh[i >> 1], dl[i >> 1]);
                }
                uint8_t *srow = smem_raw + row * 256;
                const int ch0 = (half * 64 + c) >> 3;  // 8 halves per chunk
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int at = ((ch0 + j) ^ (row & 15)) << 4;
                    *reinterpret_cast<uint4 *>(srow + at) = make_uint4(ph[4 * j], ph[4 * j + 1], ph[4 * j + 2], ph[4 * j + 3]);
                    *reinterpret_cast<uint4 *>(srow + 32768 + at) = make_uint4(pl[4 * j], pl[4 * j + 1], pl[4 * j + 2], pl[4 * j + 3]);
                    *reinterpret_cast<uint4 *>(srow + 65536 + at) = make_uint4(dh[4 * j], dh[4 * j + 1], dh[4 * j + 2], dh[4 * j + 3]);
                    *reinterpret_cast<uint4 *>(srow + 98304 + at) = make_uint4(dl[4 * j], dl[4 * j + 1], dl[4 * j + 2], dl[4 * j + 3]);
                }
            }
        }
        if (__any_sync(0xffffffffu, saturated) && lane == 0) atomicAdd(&g_tc_saturated, 1u);
        mbar_arrive_warp(&sh->staged);
        if (__all_sync(0xffffffffu, wwait(&sh->staged, 0, sh)) && !sh->abort) {
            // warp w writes rows [16 w, 16 w + 16) of each of the four tiles, two rows (512 bytes) per instruction
            const int w8 = warp - 2;
            const long long plane = (long long)p.Tp * p.Tp;
            const int ch = lane & 15;
#pragma unroll
            for (int pl4 = 0; pl4 < 4; ++pl4) {
                __half *dst = (pl4 < 2 ? p.p_planes : p.ds_planes) + ((long long)((pl4 & 1) * p.unit_cap + u)) * plane;
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    const int r = w8 * 16 + i + (lane >> 4);
                    const uint4 x = *reinterpret_cast<const uint4 *>(smem_raw + pl4 * 32768 + r * 256 + ((ch ^ (r & 15)) << 4));
                    *reinterpret_cast<uint4 *>(dst + (long long)(m0 + r) * p.Tp + n0 + ch * 8) = x;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------------------------------
// The same P and dS with the query side resident.  One CTA per (128 query rows, head): the hi planes of its Q and
// dO rows live in TMEM (128 columns each, A operands), their lo planes in shared memory (64 KB each), and the CTA
// walks the key tiles at or below its diagonal, 128 keys at a time.  K and V arrive as 64-column blocks (128 keys x
// 64 columns, hi and lo: 32 KB) through a ring of three; per key tile, S (4 blocks x 12 MMAs of N = 128) into one
// 128-column accumulator, then dP into the other.  Against bwd_wide_scores every operand byte of the query side
// is loaded once per CTA instead of once per tile: half the traffic from L2, which is what bounds both.
// The sixteen row warps, a thread per query row and 32 of the tile's keys, read S as soon as it is complete (P, kept in registers, goes to memory while dP's
// MMAs run), then dP (dS goes out while the next tile's S runs): the accumulators are single, and free again as
// soon as they have been read.  No shared memory is left for staging rows, so a tile's rows reach memory from
// registers: four lanes exchange 4 x 4 blocks of 16-byte chunks, and an instruction writes 64-byte runs of 8 rows.
// grid (units of the chunk, query tiles), 576 threads.
// With eight row warps of 64 keys a thread their splitting and storing, in series between S and dP, was longer than a tile's MMAs:
// us, eight -> sixteen, one sequence of T 700, 8/2 heads of 160 48 -> 39; 2 of T 3000, 16/4 of 192 594 -> 521; batch 8, T 1024,
// 32/8 of 256 623 -> 606 (the planes' DRAM traffic next).
// ---------------------------------------------------------------------------------------------------
struct ResShared {
    uint64_t full[4], freed[4], qh_full, ql_full, a_ready, s_full, s_free, dp_full, dp_free;
    uint32_t tmem_base;
    volatile int abort;
};
__device__ __forceinline__ bool rwait(uint64_t *bar, uint32_t parity, ResShared *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}
__device__ __forceinline__ void rgive_up(ResShared *sh, int code) {
    sh->abort = code;
    atomicMax(&g_tc_status, code);
}
// 16 packed words (32 halves, four 16-byte chunks) of this thread's row -> global memory: the four lanes of a quad
// exchange chunks so that lane j holds chunk j of the quad's four rows, and each of the four stores below writes
// 64 contiguous bytes of 8 rows.  `dst` points at the chunk-0 position of the quad's FIRST row; rows are `ld`
// halves apart.
__device__ __forceinline__ void store_rows_quad(__half *dst, long long ld, const uint32_t (&w)[16], int lane) {
    uint32_t r[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = w[i];
#pragma unroll
    for (int M = 2; M >= 1; M >>= 1) {
        const bool up = (lane & M) != 0;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (m & M) continue;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t send = up ? r[4 * m + e] : r[4 * (m ^ M) + e];
                const uint32_t recv = __shfl_xor_sync(0xffffffffu, send, M);
                if (up) r[4 * m + e] = recv;
                else r[4 * (m ^ M) + e] = recv;
            }
        }
    }
    // r[4 i .. 4 i + 3] = chunk (lane & 3) of the quad's row i
    const int j = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4 *>(dst + i * ld + j * 8) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
}

// Slots of the ring of K and V blocks: what shared memory leaves beside the lo planes of Q and dO.
template <int D>
__host__ __device__ constexpr int res_slots() { return D == 256 ? 3 : 4; }

template <int D>
__global__ void __launch_bounds__(kResThreads, 1)
    bwd_wide_scores_res(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                        const __grid_constant__ CUtensorMap gmap, const __grid_constant__ CUtensorMap vmap, const WideParams p) {
    constexpr int NB = D / 64, NR = res_slots<D>();
    constexpr int BT = 128 * 64 * 2;          // one 64-column block of a 128-row tile, one plane: 16 KB
    constexpr int cQh = 0, cGh = 128, cS = 256, cDP = 384;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *sQl = smem_raw, *sGl = smem_raw + NB * BT;   // lo planes of Q and dO: NB blocks each (hi planes first, staged)
    uint8_t *ring = smem_raw + 2 * NB * BT;                   // slot s: block hi, block lo at ring + s * 2 BT + {0, 1} BT
    ResShared *sh = reinterpret_cast<ResShared *>(ring + NR * 2 * BT);
    const int warp = threadIdx.x >> 5;
    // launch order (x fastest): every unit's last query tile, then every unit's last but one, ...: the longest
    // walks of the whole launch start first, so its tail is a fraction of a short walk
    const int m = (int)gridDim.y - 1 - (int)blockIdx.y;
    const int m0 = m * 128;
    const int u = (int)blockIdx.x, ug = p.unit0 + u;
    const int b = ug / p.n_heads, h = ug % p.n_heads;
    const int group = p.n_heads / p.n_kv_heads, g = h / group;
    const int B = p.batch;
    const int n_tiles = m + 1;
    const int n_blocks = 2 * NB * n_tiles;  // per tile: K's blocks, then V's

    if (threadIdx.x == 0) {
        for (int i = 0; i < NR; ++i) mbar_init(&sh->full[i], 1), mbar_init(&sh->freed[i], 1);
        mbar_init(&sh->qh_full, 1), mbar_init(&sh->ql_full, 1);
        mbar_init(&sh->a_ready, 16);
        mbar_init(&sh->s_full, 1), mbar_init(&sh->s_free, 16);
        mbar_init(&sh->dp_full, 1), mbar_init(&sh->dp_free, 16);
        sh->abort = (smem_u32(smem_raw) & 1023u) ? 90 : 0;
        if (sh->abort) atomicMax(&g_tc_status, 90);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&sh->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait();
    pdl_launch();

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one() && !sh->abort) {
            tma_prefetch_desc(&qmap), tma_prefetch_desc(&kmap), tma_prefetch_desc(&gmap), tma_prefetch_desc(&vmap);
            // the hi planes first, into the lo planes' place, until the row threads have moved them to TMEM
            mbar_arrive_expect_tx(&sh->qh_full, 2 * NB * BT);
            for (int blk = 0; blk < NB; ++blk) {
                tma_load_4d(sQl + blk * BT, &qmap, &sh->qh_full, 0, m0, h * NB + blk, b);
                tma_load_4d(sGl + blk * BT, &gmap, &sh->qh_full, 0, m0, h * NB + blk, b);
            }
            int issued = 0;
            bool live = true;
            auto load_block = [&](int j) {
                const int st = j % NR;
                if (j >= NR && !rwait(&sh->freed[st], (uint32_t)(((j / NR) & 1) ^ 1), sh)) { rgive_up(sh, 91), live = false; return; }
                const int n = j / (2 * NB), in_tile = j - n * 2 * NB;
                const bool is_v = in_tile >= NB;
                const int blk = is_v ? in_tile - NB : in_tile;
                const CUtensorMap *mp = is_v ? &vmap : &kmap;
                uint8_t *base = ring + st * 2 * BT;
                mbar_arrive_expect_tx(&sh->full[st], 2 * BT);
                tma_load_4d(base, mp, &sh->full[st], 0, n * 128, g * NB + blk, b);
                tma_load_4d(base + BT, mp, &sh->full[st], 0, n * 128, g * NB + blk, B + b);
                ++issued;
            };
            for (int j = 0; j < NR && j < n_blocks; ++j) load_block(j);
            if (!rwait(&sh->a_ready, 0, sh)) rgive_up(sh, 91), live = false;
            if (live) {
                mbar_arrive_expect_tx(&sh->ql_full, 2 * NB * BT);
                for (int blk = 0; blk < NB; ++blk) {
                    tma_load_4d(sQl + blk * BT, &qmap, &sh->ql_full, 0, m0, h * NB + blk, B + b);
                    tma_load_4d(sGl + blk * BT, &gmap, &sh->ql_full, 0, m0, h * NB + blk, B + b);
                }
            }
            for (int j = NR; live && j < n_blocks; ++j) load_block(j);
            if (sh->abort) {
                mbar_wait(&sh->qh_full, 0);
                if (live) mbar_wait(&sh->ql_full, 0);
                for (int j = (issued > NR ? issued - NR : 0); j < issued; ++j) mbar_wait(&sh->full[j % NR], (uint32_t)((j / NR) & 1));
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_f16(128, 128, false, false);
            const int steps = head_steps(p.dim_out);
            bool ok = !sh->abort && rwait(&sh->a_ready, 0, sh) && rwait(&sh->ql_full, 0, sh);
            if (!ok) rgive_up(sh, 92);
            tc_fence_after();
            const uint32_t ring_u32 = smem_u32(ring);
            const uint32_t ql_u32 = smem_u32(sQl), gl_u32 = smem_u32(sGl);
            int j = 0;  // ring block counter
            for (int n = 0; ok && n < n_tiles; ++n) {
                for (int prod = 0; ok && prod < 2; ++prod) {  // 0: S = Q K^T, 1: dP = dO V^T
                    // the accumulator must have been read by the row threads (tile n-1)
                    if (n >= 1 && !rwait(prod ? &sh->dp_free : &sh->s_free, (uint32_t)((n - 1) & 1), sh)) { rgive_up(sh, 93); ok = false; break; }
                    tc_fence_after();
                    const uint32_t acc = tmem + (prod ? cDP : cS), a_hi = tmem + (prod ? cGh : cQh);
                    const uint32_t a_lo = prod ? gl_u32 : ql_u32;
                    for (int blk = 0; blk < NB; ++blk, ++j) {
                        const int st = j % NR;
                        if (!rwait(&sh->full[st], (uint32_t)((j / NR) & 1), sh)) { rgive_up(sh, 94); ok = false; break; }
                        tc_fence_after();
                        const uint32_t base = ring_u32 + (uint32_t)(st * 2 * BT);
                        const uint64_t bh = desc_kmajor(base), bl = desc_kmajor(base + BT);
                        const uint64_t al = desc_kmajor(a_lo + (uint32_t)(blk * BT));
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            if (blk * 4 + kk >= steps) break;
                            const uint64_t dbh = desc_advance(bh, kk * 32), dbl = desc_advance(bl, kk * 32);
                            const uint32_t at = a_hi + (uint32_t)((blk * 4 + kk) * 8);
                            mma_ts_f16(acc, at, dbh, idesc, (blk > 0 || kk > 0) ? 1 : 0);
                            mma_ts_f16(acc, at, dbl, idesc, 1);
                            mma_ss_f16(acc, desc_advance(al, kk * 32), dbh, idesc, 1);
                        }
                        mma_commit(&sh->freed[st]);
                    }
                    if (ok) mma_commit(prod ? &sh->dp_full : &sh->s_full);
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ a thread per query row and 32 of the tile's 128 keys
        const int lane = threadIdx.x & 31;
        const int lane_grp = warp & 3;
        const int quarter = (warp - 2) >> 2;
        const int row = lane_grp * 32 + lane;
        const uint32_t lane_base = (uint32_t)(lane_grp * 32) << 16;
        const int t = m0 + row;
        bool ok = true;
        {
            // this row's hi plane of Q (even quarters) or of dO (odd ones), every other block of it, -> TMEM, out of the 128-byte-swizzled staging tiles
            if (!__all_sync(0xffffffffu, rwait(&sh->qh_full, 0, sh))) rgive_up(sh, 95), ok = false;
            const uint8_t *src = (quarter & 1 ? sGl : sQl) + row * 128;
#pragma unroll 1
            for (int blk = quarter >> 1; blk < NB; blk += 2) {
                uint32_t r[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 v4 = *reinterpret_cast<const uint4 *>(src + blk * BT + ((c ^ (row & 7)) << 4));
                    r[4 * c] = v4.x, r[4 * c + 1] = v4.y, r[4 * c + 2] = v4.z, r[4 * c + 3] = v4.w;
                }
                tmem_st32(tmem + lane_base + (quarter & 1 ? cGh : cQh) + blk * 32, r);
            }
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive_warp(&sh->a_ready);
        }
        const int bg = b * p.n_kv_heads + g;
        const float mq = block_mult(p.amax_q[bg]), mk = block_mult(p.amax_k[bg]);
        const float mv = block_mult(p.amax_v[bg]), mdo = block_mult(p.amax_do[bg]);
        const long long ridx = ((long long)b * p.T + (t < p.T ? t : 0)) * p.n_heads + h;
        float cq = 1.f, rel = 1.f;
        if (t < p.T) ds_row_scale(__ldg(p.rnorm + ridx), p.rnmax[bg], p.vnmax[bg], cq, rel);
        const float cs = p.scale_log2 / (mq * mk);
        const float lse2 = (t < p.T) ? __ldg(p.lse + ridx) * kLog2e - log2f(p.p_scale) : 0.f;
        const float c1 = cq / (mdo * mv * p.p_scale);
        const float dels = (t < p.T && !ZT_DEFECT(13)) ? __ldg(p.delta + ridx) * cq / p.p_scale : 0.f;
        float ds_top = 0.f;
        const long long plane = (long long)p.Tp * p.Tp;
        // the quad's first row, this thread's 32 columns, of the unit's hi planes (lo: unit_cap planes further)
        __half *p_hi = p.p_planes + (long long)u * plane + (long long)(m0 + (row & ~3)) * p.Tp + quarter * 32;
        __half *d_hi = p.ds_planes + (long long)u * plane + (long long)(m0 + (row & ~3)) * p.Tp + quarter * 32;
        const long long lo_off = (long long)p.unit_cap * plane;
        for (int n = 0; ok && n < n_tiles; ++n) {
            const int n0 = n * 128;
            const bool diag = (n == m) || (m0 + 128 > p.T);
            float2 pr[16];
            if (!__all_sync(0xffffffffu, rwait(&sh->s_full, (uint32_t)(n & 1), sh))) { rgive_up(sh, 96); ok = false; break; }
            tc_fence_after();
            {
                uint32_t rs[32];
                tmem_ld32(tmem + lane_base + cS + quarter * 32, rs);
                tmem_wait_ld();
                // S has been read: the next tile's may overwrite it
                tc_fence_before();
                mbar_arrive_warp_relaxed(&sh->s_free);
                const int key0 = n0 + quarter * 32;
                uint32_t ph[16], pl[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 x = fma2(floats2(rs[2 * i], rs[2 * i + 1]), make_float2(cs, cs), make_float2(-lse2, -lse2));
                    pr[i] = make_float2(ex2(x.x), ex2(x.y));
                }
                if (diag) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const auto vis = [&](int key) { return (key <= t || ZT_DEFECT(11)) && key < p.T && t < p.T; };
                        pr[i].x = vis(key0 + 2 * i) ? pr[i].x : 0.f, pr[i].y = vis(key0 + 2 * i + 1) ? pr[i].y : 0.f;
                    }
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) split_pack(pr[i], ph[i], pl[i]);
                store_rows_quad(p_hi + n0, p.Tp, ph, lane);
                store_rows_quad(p_hi + lo_off + n0, p.Tp, pl, lane);
            }
            if (!__all_sync(0xffffffffu, rwait(&sh->dp_full, (uint32_t)(n & 1), sh))) { rgive_up(sh, 97); ok = false; break; }
            tc_fence_after();
            {
                uint32_t rd[32];
                tmem_ld32(tmem + lane_base + cDP + quarter * 32, rd);
                tmem_wait_ld();
                tc_fence_before();
                mbar_arrive_warp_relaxed(&sh->dp_free);
                uint32_t dh[16], dl[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    // (pr is zero where masked)
                    float2 x = mul2(pr[i], fma2(floats2(rd[2 * i], rd[2 * i + 1]), make_float2(c1, c1), make_float2(-dels, -dels)));
                    x.x = clamp_abs(x.x, kDsBound), x.y = clamp_abs(x.y, kDsBound);
                    ds_top = max3(ds_top, fabsf(x.x), fabsf(x.y));
                    split_pack(x, dh[i], dl[i]);
                }
                store_rows_quad(d_hi + n0, p.Tp, dh, lane);
                store_rows_quad(d_hi + lo_off + n0, p.Tp, dl, lane);
            }
        }
        if (__any_sync(0xffffffffu, ds_top >= kDsBound) && lane == 0) atomicAdd(&g_tc_saturated, 1u);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}
template <int D>
inline size_t res_smem_bytes() { return (size_t)(2 * D / 64 + 2 * res_slots<D>()) * (128 * 64 * 2) + sizeof(ResShared); }

// ---------------------------------------------------------------------------------------------------
// The three products that read the planes, in one launch of persistent blocks.  128 x 256 output tiles (a head's whole
// width, so that a tile of the planes is read once), 64-deep steps, B always the tensor whose rows are the contraction
// index ([T, width] planes read as N-major tiles).  (128 x 192 tiles, where the planes are 192 columns wide a head.)
//   dQ      A = dS planes, K-major; contraction over keys [piece * 1024, min((m + 1) * 128, (piece + 1) * 1024)); row t leaves
//           times scale / (cq(t) mk).
//   dK, dV  A = dS or P planes read M-major (rows are the contraction index: query rows); contraction over query rows
//           [max(m * 128, piece * 1024), min(Tp, (piece + 1) * 1024)); every head of a group adds into its KV head.
// dQ's tiles are stored where one unit holds a tile's whole contraction (T up to 1024); every other tile is added to the output
// (red.global.add.v4.f32), which the pre-pass has zeroed.
// A unit is one (product, head of the chunk, piece, tile): nine steps of MMAs on average at T 1024, about as long as its
// prologue and epilogue together when each was a block of its own.  So a block walks its share of the units with two
// accumulators in TMEM (all 512 columns), loads run ahead across units, and a unit's epilogue -- straight from TMEM to
// memory, rows regrouped among eight lanes -- runs under the next one's MMAs.  A head's tiles are consecutive units:
// blocks that run together share its operands in L2.  Where a tile is one unit (T up to 1024) and
// products_in_turn allows it, so are those of its three products, in turn, and dS is still in L2 when the second of its two products reads it;
// longest first, and the other way round in every second head, so that what a block gets by its stride is neither always long nor
// always short.  (With pieces this was 5 % slower, T 3000: 789 -> 827.)  Batch 8, T 1024, 32/8 heads of 256, in the order of the
// products / in turn: 773 / 702 (and 785 with dQ added instead of stored).
// Us, three launches of a block per unit -> this: batch 8, T 1024, 32/8 heads of 256 809 -> 777 (bound by DRAM: the planes are
// 3 GB written and read there); forward and backward at batch 4, T 300, 8/2 heads 129 -> 111, one sequence of T 500, 4/2
// heads of 160 130 -> 102.
// ---------------------------------------------------------------------------------------------------
struct TriShared {
    uint64_t full[2], freed[2], acc_full[2], acc_free[2];
    uint32_t tmem_base;
    volatile int abort;
};
__device__ __forceinline__ bool twait(uint64_t *bar, uint32_t parity, TriShared *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}
__device__ __forceinline__ void tgive_up(TriShared *sh, int code) {
    sh->abort = code;
    atomicMax(&g_tc_status, code);
}
// Whether a head's units of the three products go in turn: where no block gets much more than the others.  The units repeat every two
// heads, 6 nt of them; a block finds its next one `blocks` further on, which moves its place in that period by `drift`, so few
// rounds leave it among the long ones (T 1024, 36 heads on 148 blocks: 25 % above the order of the products), and it is as good once
// they have gone through three fifths of the period.  Us, in the order of the products / in turn, heads of 192 and of 256 columns:
// T 1024, 16 heads 53.8 / 61.2 and 62 / 71, 32 88.5 / 91.6 and 99 / 101, 64 156 / 154 and 191 / 188, 256 637 / 560 and 773 / 702; T 500, 32
// 32.4 / 35.2 and 38.2 / 41.5, 64 59.5 / 55.9 and 70.8 / 67.0.
__host__ __device__ inline bool products_in_turn(int pieces, int nt, int heads, int blocks) {
    const int place = blocks % (6 * nt), drift = place < 6 * nt - place ? place : 6 * nt - place;
    return pieces == 1 && 5LL * heads * drift >= 6LL * blocks;
}

struct TriUnit {
    int which, u, m0, b, h, k_begin, n_steps;  // which: 0 dQ, 1 dK, 2 dV; n_steps <= 0: nothing to do
    __host__ __device__ __forceinline__ TriUnit(const WideParams &p, int i) {
        const int nt = p.Tp / 128;
        int m, piece = 0;
        if (p.in_turn) {
            u = i / (3 * nt);
            const int at = i - u * 3 * nt, r = u & 1 ? 3 * nt - 1 - at : at, level = r / 3;
            which = r - 3 * level;
            m = which == 0 ? nt - 1 - level : level;
        } else {
            const int r = i / nt % (p.units * p.pieces);
            which = i / (nt * p.units * p.pieces);
            m = i % nt, u = r / p.pieces, piece = r - u * p.pieces;
        }
        const int ug = p.unit0 + u;
        b = ug / p.n_heads, h = ug - b * p.n_heads;
        m0 = m * 128;
        k_begin = piece * kPiece;
        int k_end = k_begin + kPiece;
        if (which == 0) k_end = k_end < m0 + 128 ? k_end : m0 + 128;
        else k_begin = k_begin > m0 ? k_begin : m0;
        k_end = k_end < p.Tp ? k_end : p.Tp;
        n_steps = (k_end - k_begin) / 64;
    }
};

template <int D>
__global__ void __launch_bounds__(kTriThreads, 1)
    wide_products(const __grid_constant__ CUtensorMap ds_k, const __grid_constant__ CUtensorMap ds_m, const __grid_constant__ CUtensorMap p_m,
                  const __grid_constant__ CUtensorMap k_n, const __grid_constant__ CUtensorMap qs_n, const __grid_constant__ CUtensorMap g_n,
                  const WideParams p, int n_units) {
    // a stage: A hi, A lo (128 x 64 halves each) and B hi, B lo (64 contraction rows x D columns each, in
    // 64-column blocks of 8 KB): 96 KB at D = 256; two stages
    constexpr int kBT = 64 * D * 2, kStage = 2 * kTB + 2 * kBT;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    TriShared *sh = reinterpret_cast<TriShared *>(smem_raw + 2 * kStage);
    const int warp = threadIdx.x >> 5;
    const int group = p.n_heads / p.n_kv_heads;
    const int B = p.batch;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh->full[i], 1), mbar_init(&sh->freed[i], 1);
            mbar_init(&sh->acc_full[i], 1), mbar_init(&sh->acc_free[i], 4);
        }
        sh->abort = (smem_u32(smem_raw) & 1023u) ? 84 : 0;
        if (sh->abort) atomicMax(&g_tc_status, 84);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&sh->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait();
    pdl_launch();

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one() && !sh->abort) {
            tma_prefetch_desc(&ds_k), tma_prefetch_desc(&ds_m), tma_prefetch_desc(&p_m);
            tma_prefetch_desc(&k_n), tma_prefetch_desc(&qs_n), tma_prefetch_desc(&g_n);
            int it = 0;  // steps issued
            for (int i = blockIdx.x; i < n_units && !sh->abort; i += gridDim.x) {
                const TriUnit w(p, i);
                const CUtensorMap *am = w.which == 0 ? &ds_k : w.which == 1 ? &ds_m : &p_m;
                const CUtensorMap *bm = w.which == 0 ? &k_n : w.which == 1 ? &qs_n : &g_n;
                // B's column blocks: the head's (dQ: the KV head's) columns
                const int bblk = (w.which == 0 ? w.h / group : w.h) * (D / 64);
                for (int s = 0; s < w.n_steps; ++s, ++it) {
                    const int st = it & 1, k0 = w.k_begin + s * 64;
                    if (it >= 2 && !twait(&sh->freed[st], (uint32_t)(((it >> 1) & 1) ^ 1), sh)) { tgive_up(sh, 85); break; }
                    uint8_t *base = smem_raw + st * kStage;
                    mbar_arrive_expect_tx(&sh->full[st], kStage);
                    // dK, dV: 64 query rows x two 64-key blocks; dQ: 128 query rows x one block
                    const int c1 = w.which ? k0 : w.m0, c2 = (w.which ? w.m0 : k0) / 64;
                    tma_load_4d(base, am, &sh->full[st], 0, c1, c2, w.u);
                    tma_load_4d(base + kTB, am, &sh->full[st], 0, c1, c2, p.unit_cap + w.u);
                    tma_load_4d(base + 2 * kTB, bm, &sh->full[st], 0, k0, bblk, w.b);
                    tma_load_4d(base + 2 * kTB + kBT, bm, &sh->full[st], 0, k0, bblk, B + w.b);
                }
            }
            if (sh->abort)
                for (int s = (it > 2 ? it - 2 : 0); s < it; ++s) mbar_wait(&sh->full[s & 1], (uint32_t)((s >> 1) & 1));
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one() && !sh->abort) {
            const uint32_t s_u32 = smem_u32(smem_raw);
            int it = 0, n = 0;  // steps, units with something to do
            for (int i = blockIdx.x; i < n_units && !sh->abort; i += gridDim.x) {
                const TriUnit w(p, i);
                if (w.n_steps <= 0) continue;
                const uint32_t idesc = idesc_f16(128, 16 * head_steps(p.dim_out), w.which != 0, true);
                const uint32_t a_step = w.which ? 2048 : 32;
                const uint32_t acc = tmem + (n & 1) * 256;
                if (n >= 2 && !twait(&sh->acc_free[n & 1], (uint32_t)(((n >> 1) & 1) ^ 1), sh)) { tgive_up(sh, 86); break; }
                for (int s = 0; s < w.n_steps; ++s, ++it) {
                    const int st = it & 1;
                    if (!twait(&sh->full[st], (uint32_t)((it >> 1) & 1), sh)) { tgive_up(sh, 86); break; }
                    tc_fence_after();
                    const uint32_t base = s_u32 + (uint32_t)(st * kStage);
                    const uint64_t ah = w.which ? desc_mnmajor_16b(base, 64 * 128) : desc_kmajor(base);
                    const uint64_t al = w.which ? desc_mnmajor_16b(base + kTB, 64 * 128) : desc_kmajor(base + kTB);
                    const uint64_t bh = desc_mnmajor_16b(base + 2 * kTB, 64 * 128);
                    const uint64_t bl = desc_mnmajor_16b(base + 2 * kTB + kBT, 64 * 128);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        const uint64_t dah = desc_advance(ah, kk * a_step), dal = desc_advance(al, kk * a_step);
                        const uint64_t dbh = desc_advance(bh, kk * 2048), dbl = desc_advance(bl, kk * 2048);
                        mma_ss_f16(acc, dah, dbh, idesc, (s > 0 || kk > 0) ? 1 : 0);
                        mma_ss_f16(acc, dah, dbl, idesc, 1);
                        mma_ss_f16(acc, dal, dbh, idesc, 1);
                    }
                    mma_commit(&sh->freed[st]);
                }
                mma_commit(&sh->acc_full[n & 1]);
                ++n;
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue: a thread per output row
        const int lane = threadIdx.x & 31, j8 = lane & 7;
        const int lane_grp = warp & 3;
        const uint32_t lane_base = (uint32_t)(lane_grp * 32) << 16;
        int n = 0;
        for (int i = blockIdx.x; i < n_units; i += gridDim.x) {
            const TriUnit w(p, i);
            if (w.n_steps <= 0) continue;
            const int g = w.h / group, bg = w.b * p.n_kv_heads + g;
            const int t = w.m0 + lane_grp * 32 + lane;  // dQ: the query row; dK, dV: the key
            float f;
            if (w.which == 0) {
                float cq = 1.f, rel = 1.f;
                if (t < p.T) ds_row_scale(__ldg(p.rnorm + ((long long)w.b * p.T + t) * p.n_heads + w.h), p.rnmax[bg], p.vnmax[bg], cq, rel);
                f = p.scale / (cq * block_mult(p.amax_k[bg]));
            } else if (w.which == 1) {
                f = p.scale / (ds_group_scale(p.rnmax[bg], p.vnmax[bg]) * block_mult(p.amax_q[bg]));
            } else {
                f = 1.0f / (p.p_scale * block_mult(p.amax_do[bg]));
            }
            if (!__all_sync(0xffffffffu, twait(&sh->acc_full[n & 1], (uint32_t)((n >> 1) & 1), sh))) { tgive_up(sh, 87); break; }
            tc_fence_after();
            const long long ld = (long long)(w.which == 0 ? p.n_heads : p.n_kv_heads) * p.dim_out;
            const int row0 = t - j8;  // the first of this lane's eight rows
            const bool whole = w.which == 0 && p.pieces == 1;
            float *dst = (w.which == 0 ? p.dq : w.which == 1 ? p.dk : p.dv) + ((long long)w.b * p.T + row0) * ld +
                         (long long)(w.which == 0 ? w.h : g) * p.dim_out + 4 * j8;
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                uint32_t r[32];
                tmem_ld32(tmem + lane_base + (n & 1) * 256 + c, r);
                tmem_wait_ld();
                if (c + 32 == D) {  // all read: the MMAs may have the buffer while the last columns are on their way
                    tc_fence_before();
                    mbar_arrive_warp_relaxed(&sh->acc_free[n & 1]);
                }
                if (c >= p.dim_out) continue;
#pragma unroll
                for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * f);
                // eight lanes transpose their 8 x 8 blocks of float4: lane j gets the j-th float4 of eight rows, and an
                // instruction covers four rows' 128-byte runs
#pragma unroll
                for (int M = 4; M >= 1; M >>= 1) {
                    const bool up = (lane & M) != 0;
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        if (m & M) continue;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint32_t send = up ? r[4 * m + e] : r[4 * (m ^ M) + e];
                            const uint32_t recv = __shfl_xor_sync(0xffffffffu, send, M);
                            if (up) r[4 * m + e] = recv;
                            else r[4 * (m ^ M) + e] = recv;
                        }
                    }
                }
                if (c + 4 * j8 < p.dim_out) {  // (a padded tile's upper columns are not the tensor's)
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        if (row0 + e >= p.T) continue;
                        const float4 a = make_float4(__uint_as_float(r[4 * e]), __uint_as_float(r[4 * e + 1]), __uint_as_float(r[4 * e + 2]), __uint_as_float(r[4 * e + 3]));
                        if (whole) *reinterpret_cast<float4 *>(dst + (long long)e * ld + c) = a;
                        else tcb::red_add_v4(dst + (long long)e * ld + c, a);
                    }
                }
            }
            ++n;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

template <int D>
inline size_t tri_smem_bytes() { return (size_t)2 * (2 * kTB + 2 * 64 * D * 2) + sizeof(TriShared); }

// ---- host side ----------------------------------------------------------------------------------------

constexpr size_t kScratchBudget = (size_t)2 << 30;   // planes of P and dS held at once, unless one KV group needs more
constexpr size_t kScratchLimit = (size_t)16 << 30;   // one KV group's planes beyond this: the shape is not taken

struct WideWorkspace {
    tcb::BwdWorkspace base;   // the fused backward's layout first: the forward may have left q, k, v planes there
    __half *p_planes, *ds_planes;  // where base has its partial results: a forward has put those together by then
    int Tp, unit_cap;
    size_t total_bytes;
};

inline int wide_unit_cap(int batch, int T, int n_heads, int n_kv_heads) {
    const long long Tp = (T + 127) / 128 * 128;
    const size_t unit = (size_t)8 * Tp * Tp;  // four planes of Tp x Tp halves
    const int group = n_heads / n_kv_heads;
    if (unit * group > kScratchLimit) return 0;
    long long cap = (long long)(kScratchBudget / unit) / group * group;
    if (cap < group) cap = group;
    const long long all = (long long)batch * n_heads;
    return (int)(cap < all ? cap : all);
}

// The layout in a workspace of `bytes`: a chunk takes as many heads as fit, one KV group's at least.
inline WideWorkspace wide_workspace(void *ws, size_t bytes, int batch, int T, int n_heads, int n_kv_heads, int td) {
    WideWorkspace w{};
    w.base = tcb::bwd_workspace(ws, batch, T, n_heads, n_kv_heads, td);
    const int group = n_heads / n_kv_heads;
    w.Tp = (T + 127) / 128 * 128;
    w.unit_cap = wide_unit_cap(batch, T, n_heads, n_kv_heads);
    const size_t half = (size_t)2 * w.Tp * w.Tp * sizeof(__half);  // P's two planes of a head, or dS's (a multiple of 64 KB)
    const size_t fit = bytes > w.base.base_bytes ? (bytes - w.base.base_bytes) / (2 * half) / group * group : 0;
    if (fit < (size_t)w.unit_cap) w.unit_cap = fit < (size_t)group ? group : (int)fit;
    char *c = static_cast<char *>(ws);
    w.p_planes = reinterpret_cast<__half *>(c + w.base.base_bytes);
    w.ds_planes = reinterpret_cast<__half *>(c + w.base.base_bytes + w.unit_cap * half);
    w.total_bytes = w.base.base_bytes + 2 * w.unit_cap * half;
    if (w.total_bytes < w.base.total_bytes) w.total_bytes = w.base.total_bytes;
    return w;
}

inline bool tc_bwd_wide_supported(int batch, int T, int n_heads, int n_kv_heads, int dim, const void *q, const void *k,
                                  const void *v, const void *dout, const void *dq, const void *dk, const void *dv) {
    if (!tc_takes_dim(dim) || dim <= 128 || T < 1 || batch < 1) return false;
    if (wide_unit_cap(batch, T, n_heads, n_kv_heads) == 0) return false;
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (!al(q) || !al(k) || !al(v) || !al(dout) || !al(dq) || !al(dk) || !al(dv)) return false;
    const DeviceInfo *d = device_info();
    return d && d->cc_major == 10 && get_encode_tiled() != nullptr;
}

inline size_t wide_smem_bytes() { return (size_t)kStages * kSB + sizeof(WideShared); }

}  // namespace tcw

// What the backward above 128 columns wants, must have, and can want at this shape or a shorter one (all 0: not taken).
inline WorkspaceNeed tc_bwd_wide_workspace_need(int batch, int T, int n_heads, int n_kv_heads, int dim) {
    if (tcw::wide_unit_cap(batch, T, n_heads, n_kv_heads) == 0) return {0, 0, 0};
    const int td = tc_tile_dim(dim), group = n_heads / n_kv_heads;
    const tcw::WideWorkspace w = tcw::wide_workspace(nullptr, SIZE_MAX, batch, T, n_heads, n_kv_heads, td);
    const size_t unit = (size_t)8 * w.Tp * w.Tp, all = unit * batch * n_heads;
    size_t planes = unit * group > tcw::kScratchBudget ? unit * group : tcw::kScratchBudget;
    if (planes > all) planes = all;
    const size_t parts = (fwd_parts_floats_bound(td) * sizeof(float) + 1023) / 1024 * 1024;
    return {w.base.base_bytes + unit * group, w.total_bytes, w.base.base_bytes + (planes > parts ? planes : parts)};
}

// delta (= sum_j dout out, per row) is formed here; dq, dk, dv are assigned.  `out` may alias dq: it has been read when
// dq is first written.
inline int launch_bwd_wide(const float *q, const float *k, const float *v, const float *out, const float *dout,
                           const float *lse, float *delta, float *dq, float *dk, float *dv, void *workspace, size_t workspace_bytes, int batch, int T,
                           int n_heads, int n_kv_heads, int dim, cudaStream_t stream, bool qkv_planes_kept = false,
                           bool tile_scores = false) {
    using namespace tcb;
    using namespace tcw;
    const int td = tc_tile_dim(dim);
    const WideWorkspace ww = wide_workspace(workspace, workspace_bytes, batch, T, n_heads, n_kv_heads, td);
    const BwdWorkspace &w = ww.base;
    const int group = n_heads / n_kv_heads;
    const int wq = n_heads * td, wkv = n_kv_heads * td;
    PassArgs pa{};
    pa.dim = dim, pa.pd = td;
    uint32_t *rnmax = w.dsmax;  // (the header's last array)
    {
        PassTensor &t = pass_add(pa, dout, batch, T, n_heads, group, w.part[3], w.amax_do, rnmax, w.do_planes);
        t.o = out, t.delta = delta, t.rnorm = w.rnorm;
    }
    pass_add(pa, q, batch, T, n_heads, group, w.part[0], w.amax_q, nullptr, w.q_planes);
    if (!qkv_planes_kept) {
        pass_add(pa, k, batch, T, n_kv_heads, 1, w.part[1], w.amax_k, nullptr, w.k_planes);
        pass_add(pa, v, batch, T, n_kv_heads, 1, w.part[2], w.amax_v, w.vnmax, w.v_planes);
    }
    const int pieces = (ww.Tp + kPiece - 1) / kPiece;
    if (pieces > 1) pass_fill(pa, dq, (long long)batch * T * n_heads * dim);  // (a whole contraction's dQ is stored)
    pass_fill(pa, dk, (long long)batch * T * n_kv_heads * dim);
    pass_fill(pa, dv, (long long)batch * T * n_kv_heads * dim);
    if (launch_pass_backward(pa, w, true, true, qkv_planes_kept, stream)) return 1;
    const int Tp = ww.Tp, cap = ww.unit_cap;
    CUtensorMap q_k, k_k, g_k, v_k;      // K-major 128-row tiles of one 64-column block: the scores' operands
    CUtensorMap k_n, qs_n, g_n;          // N-major tiles (64 contraction rows x the head's 256 columns): B of the three products
    CUtensorMap ds_k, ds_m, p_m;         // the planes: K-major A (dQ), M-major A (dK, dV)
    if (!make_half_tile_map(&q_k, w.q_planes, 2 * batch, T, wq, 64, 128) ||
        !make_half_tile_map(&k_k, w.k_planes, 2 * batch, T, wkv, 64, 128) ||
        !make_half_tile_map(&g_k, w.do_planes, 2 * batch, T, wq, 64, 128) ||
        !make_half_tile_map(&v_k, w.v_planes, 2 * batch, T, wkv, 64, 128) ||
        !make_half_tile_map(&k_n, w.k_planes, 2 * batch, T, wkv, td, 64) ||
        !make_half_tile_map(&qs_n, w.qs_planes, 2 * batch, T, wq, td, 64) ||
        !make_half_tile_map(&g_n, w.do_planes, 2 * batch, T, wq, td, 64) ||
        !make_half_tile_map(&ds_k, ww.ds_planes, 2 * cap, Tp, Tp, 64, 128) ||
        !make_half_tile_map(&ds_m, ww.ds_planes, 2 * cap, Tp, Tp, 128, 64) ||
        !make_half_tile_map(&p_m, ww.p_planes, 2 * cap, Tp, Tp, 128, 64))
        return refuse("the TMA tensor maps for the wide-head backward could not be encoded.");
    const size_t smem = wide_smem_bytes();
    const size_t smem_t = td == 192 ? tri_smem_bytes<192>() : tri_smem_bytes<256>();
    const size_t smem_r = td == 192 ? res_smem_bytes<192>() : res_smem_bytes<256>();
    const auto scores = td == 192 ? bwd_wide_scores_res<192> : bwd_wide_scores_res<256>;
    const auto products = td == 192 ? wide_products<192> : wide_products<256>;
    if (optin_smem((const void *)bwd_wide_scores, smem) || optin_smem((const void *)scores, smem_r) ||
        optin_smem((const void *)products, smem_t))
        return 1;
    WideParams p{};
    p.lse = lse, p.delta = delta, p.rnorm = w.rnorm;
    p.amax_q = w.amax_q, p.amax_k = w.amax_k, p.amax_v = w.amax_v, p.amax_do = w.amax_do;
    p.vnmax = w.vnmax, p.rnmax = rnmax;
    p.p_planes = ww.p_planes, p.ds_planes = ww.ds_planes;
    p.batch = batch, p.T = T, p.Tp = Tp, p.n_heads = n_heads, p.n_kv_heads = n_kv_heads;
    p.dim_out = dim, p.td = td;
    p.unit_cap = cap;
    p.dq = dq, p.dk = dk, p.dv = dv;
    p.pieces = pieces;
    p.scale = 1.0f / sqrtf((float)dim), p.scale_log2 = kLog2e / sqrtf((float)dim);
    p.p_scale = ldexpf(1.0f, 10);
    g_last_path = "tcgen05";
    const int nt = Tp / 128;
    const int all = batch * n_heads;
    for (int unit0 = 0; unit0 < all; unit0 += cap) {
        const int units = all - unit0 < cap ? all - unit0 : cap;
        p.unit0 = unit0;
        if (tile_scores) {
            const dim3 gs((unsigned)(nt * (nt + 1) / 2), (unsigned)units);
            if (launch_after("bwd_wide_scores", bwd_wide_scores, gs, dim3(kScoreThreads), smem, stream, 1, q_k, k_k, g_k, v_k, p)) return 1;
        } else {
            const dim3 gs((unsigned)units, (unsigned)nt);
            if (launch_after("bwd_wide_scores_res", scores, gs, dim3(kResThreads), smem_r, stream, 1, q_k, k_k, g_k, v_k, p)) return 1;
        }
        p.units = units;
        const long long n_units = 3LL * nt * units * p.pieces;
        const dim3 gp((unsigned)(n_units < split_sm_count() ? n_units : split_sm_count()));
        p.in_turn = products_in_turn(p.pieces, nt, units, split_sm_count());
        if (launch_after("wide_products", products, gp, dim3(kTriThreads), smem_t, stream, 1, ds_k, ds_m, p_m, k_n, qs_n, g_n, p, (int)n_units))
            return 1;
    }
    return 0;
}

}  // namespace zt
