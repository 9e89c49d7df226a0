// Causal GQA attention forward on the tensor cores with the three-term split on f16 pieces
// (the arithmetic of tc_bwd.cuh) and a two-deep pipeline over the key tiles.
//
// Same result as attn_fwd_tc (tc_fwd.cuh, 3xTF32) and the same role -- attention.forward
// (src/attention.zig:60-153) for a batch plus each row's log-sum-exp -- at 2.4 times the speed:
// an f16 term is half a TF32 MMA, operands take half the bytes (three K and three V tiles, hi and
// lo, fit in shared memory), and two S tiles and two O accumulators fit in TMEM.
//
//   the pre-pass             (prepass.cuh) k, v -> f16 hi/lo planes with a power-of-two scale
//                            per (sequence, KV group), in a workspace.
//   TMA warp        K and V hi/lo tiles of 64 keys, a ring of three slots each: a K tile is free
//                   once its S has retired, two tiles before its V.
//   MMA warp        S[j+2] = Qh.Kh + Qh.Kl + Ql.Kh  (A = Q from TMEM) into buffer j & 1 as soon as
//                   P.V of tile j has been issued; once P[j] is in TMEM,
//                   O[j & 1] += Ph.Vh + Ph.Vl + Pl.Vh   (A = P from TMEM, V tile as MN-major B).
//   softmax warps   two sets of four, one thread per query row; set j & 1 owns tile j, with a
//                   reference maximum (moved only when it grows by > 2^8), a sum and an O accumulator
//                   of its own, so neither set waits on the other's tile.  P is scaled by 2^7 and
//                   split into packed f16 pairs written over S.  The two partial softmaxes are merged
//                   when the row is written.
// TMEM columns: [0,D/2) Qh, [D/2,D) Ql, [D,2D) O of set 0, [2D,3D) O of set 1, then two S/P tiles of
// 64 columns.
#pragma once

#include "tc_bwd.cuh"

namespace zt {
namespace tcf16 {

using namespace tc;
using tcb::block_mult;
using tcb::split_pack;
using tcb::fma2;
using tcb::add2;
using tcb::max3;
using tcb::floats2;

constexpr int kThreads = 320;  // 8 softmax warps (two sets of four), 1 TMA warp, 1 MMA warp
constexpr float kPScale = 128.0f;  // 2^7: P is multiplied by it before its 16-bit split (the 7.0f in the kernels)
constexpr float kRescaleThreshold = 8.0f;

struct Shared {
    uint64_t full_k[3], free_k[3], full_v[3], free_v[3];
    uint64_t a_ready, s_full[2], p_full[2], pv_done[2], all_done, q_full;
    uint32_t tmem_base;
    volatile int abort;
    float fin_m[2][128], fin_l[2][128];  // each set's reference maximum and sum, for the final merge
    float fin_f[2][128];                 // what has been flushed of its O is relative to this maximum (-inf: nothing)
    float q_top[2][128];                 // max |q| of each half of a row's columns
};

struct Params {
    const uint32_t *amax_k, *amax_v;            // [B, Hkv]
    uint32_t *amax_q;                           // [B, Hkv]: takes the maximum of every query row (cleared before); null: not wanted
    const float2 *rope;                         // null, or the (cos, sin) table [T][dim_out / 2] to rotate the query rows with
    float *flush_rows;                          // [B, T, H, dim_out]: where attn_fwd_tc16 keeps its second set's flushed sums
    float *out, *lse;                           // lse may be null
    int batch, T, n_heads, n_kv_heads;
    int q_offset;  // query row r stands at position q_offset + r of the keys: it sees keys 0 .. q_offset + r
    int parts;     // CTAs along a query tile's keys; with more than one, out and lse are the parts' (see tc_split.cuh):
    long long out_part, lse_part;  // elements from one part's to the next
    bool by_tile;  // (one head a block) blocks go through the sequences tile by tile, see tile_by_tile
    bool flush;    // of a window whose accumulators take more than kFlushKeyTiles key tiles: O leaves them after every so many (see flush_row)
    int dim_out;  // the tensors' head_dim, at most the tile's D
    int ahead;    // attn_fwd_tc16 prefetches the query tile of the block this many places on in launch order; 0: none
    float scale_log2;
    // When set, the epilogue also leaves out as f16 hi/lo planes ([2][B][T][H * dim_out], one power-of-two scale per
    // sequence) for the projection that follows (tc_gemm.cuh): the GEMM then needs no pass of its own over out.
    __half *o_planes;
    long long o_plane_stride;  // elements from the hi plane to the lo plane
    PeerList out_peers;        // out is also stored here (same element index), see zt_common.cuh
};

// The scale of a sequence's out planes.  An output row is a convex combination of rows of v, so |out| <= max |v|
// over the sequence's KV heads: the power of two that puts that maximum just under 2^15 fits out as well.
__device__ __forceinline__ float out_plane_mult(const Params &p, int b) {
    uint32_t top = 0;
    for (int g = 0; g < p.n_kv_heads; ++g) top = max(top, p.amax_v[b * p.n_kv_heads + g]);
    return block_mult(top);
}
// Four consecutive elements of out at element index idx, and their planes when asked for.
__device__ __forceinline__ void store_out4(const Params &p, long long idx, float4 o4, float mo) {
    *reinterpret_cast<float4 *>(p.out + idx) = o4;
    for (int r = 0; r < p.out_peers.n; ++r) *reinterpret_cast<float4 *>(p.out_peers.ptr[r] + idx) = o4;
    if (p.o_planes) {
        uint2 hw, lw;
        split_pack(o4.x * mo, o4.y * mo, hw.x, lw.x);
        split_pack(o4.z * mo, o4.w * mo, hw.y, lw.y);
        *reinterpret_cast<uint2 *>(p.o_planes + idx) = hw;
        *reinterpret_cast<uint2 *>(p.o_planes + p.o_plane_stride + idx) = lw;
    }
}

__device__ __forceinline__ bool fwait(uint64_t *bar, uint32_t parity, Shared *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}
__device__ __forceinline__ void fgive_up(Shared *sh, int code) {
    sh->abort = code;
    atomicMax(&g_tc_status, code);
}

// The row work on 32 score columns.  A softmax's warps share their schedulers' slots with each other and with the warp that issues the
// MMAs, so it is paired (f32x2, three-operand maxima): ten instructions for two columns where there were fourteen.  Us of the forward,
// before -> after: 512 rows at 3584 keys, 32/8 of
// 128 103 -> 99 (with the rows' way out, send_row).
// Columns beyond the `visible` first one take no part: a tile needs this only where it reaches beyond the first of a warp's rows.
__device__ __forceinline__ void mask32(uint32_t (&r)[32], int visible) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (i > visible) r[i] = 0xff800000u;
}
__device__ __forceinline__ float row_max32(const uint32_t (&r)[32], float m) {
    float n = -INFINITY;  // (a chain of its own)
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
        m = max3(m, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
        n = max3(n, __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
    }
    return fmaxf(m, n);
}
// P comes out already multiplied by kPScale (the scale rides in the exponent: `off` is the reference maximum minus log2 kPScale), split into
// packed f16 pairs.
__device__ __forceinline__ float row_exp32(const uint32_t (&r)[32], float cs, float off, uint32_t (&ph)[16], uint32_t (&pl)[16]) {
    const float2 cs2 = make_float2(cs, cs), off2 = make_float2(-off, -off);
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const float2 x = fma2(floats2(r[i], r[i + 1]), cs2, off2);
        const float2 pe = make_float2(ex2(x.x), ex2(x.y));
        sum = add2(sum, pe);
        split_pack(pe, ph[i >> 1], pl[i >> 1]);
    }
    return sum.x + sum.y;
}

// The tensor core adds into its f32 accumulator with truncation, which over n key tiles of 64 costs O about
// n 2.3e-7 of its size, always toward zero (1.4e-5 measured at 4096 keys in one accumulator).  With FLUSH
// O leaves TMEM every so many tiles and is summed with rounding in memory: in the row of out, which the finished row
// overwrites at the end.  16 tiles hold the error at 3.7e-6 whatever the context, for 64 KB through L2 per 32000
// clocks of MMAs.  Set for windows of a prompt, every row of which runs over the whole context behind it; over a whole
// sequence the rows that see few keys carry the result's norm.
constexpr int kFlushKeyTiles = 16;
// Four columns of the running sum: the first flush starts it, `f` moves it to the current reference maximum.
__device__ __forceinline__ float4 flush_sum4(const float *at, float f, bool first, float4 o) {
    if (first) return o;
    const float4 g = *reinterpret_cast<const float4 *>(at);
    o.x = fmaf(g.x, f, o.x), o.y = fmaf(g.y, f, o.y), o.z = fmaf(g.z, f, o.z), o.w = fmaf(g.w, f, o.w);
    return o;
}
// Where a row's running sum is kept, null when the row is not the tensor's; `width` columns of it (the rest are padding).  The sums are their
// threads' own, so a warp's lie in its rows of the tensor as they come -- the lanes' first four columns, then their next four -- and an
// instruction covers 512 bytes in a stretch or two.  (Each in its own row, an instruction touched 32 lines: 10000 clocks a flush and 17000 at a
// block's end of 143000 in all, 512 rows at 3584 keys, 32/8 heads of 128.  Us, the kernel there 93.8 -> 86.4; 2000 rows at 8000, 8/2 heads of 128
// 243 -> 200; in attn_fwd_tc16g 2048 at 2000, 32/8 of 128 297 -> 249.)
struct FlushRow {
    float *sums;  // the warp's first row
    int width, stride, rows;  // columns of a row; from a row to the next; the warp's that are the tensor's
    uint32_t per;             // 2^20 over the row's float4, rounded up: i, below 32 rows of at most 64, is divided by them exactly
    __device__ __forceinline__ float *at(int col) const {
        const int i = (col >> 2) * rows + (int)(threadIdx.x & 31), r = (int)(((uint32_t)i * per) >> 20);
        return sums + (long long)r * stride + (i - r * (width >> 2)) * 4;
    }
};
// For the warp whose rows of head h begin with t0, in `tensor` [B, T, H, dim_out].
__device__ __forceinline__ FlushRow flush_row_at(const Params &p, float *tensor, int b, int t0, int h) {
    const int rows = p.T - t0 < 32 ? p.T - t0 : 32;
    FlushRow w{nullptr, p.dim_out, p.n_heads * p.dim_out, rows, (1u << 20) / (uint32_t)(p.dim_out >> 2) + 1u};
    if ((int)(threadIdx.x & 31) < rows) w.sums = tensor + (((long long)b * p.T + t0) * p.n_heads + h) * p.dim_out;
    return w;
}
// O's columns [0, D) of this thread's row, at TMEM `taddr`, into its running sum.
template <int D>
__device__ __forceinline__ void flush_row(uint32_t taddr, const FlushRow &row, float f, bool first) {
#pragma unroll 1
    for (int c = 0; c < D; c += 32) {
        uint32_t r[32];
        tmem_ld32(taddr + c, r);
        tmem_wait_ld();
        if (row.sums == nullptr) continue;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            if (c + i >= row.width) break;
            float *at = row.at(c + i);
            *reinterpret_cast<float4 *>(at) = flush_sum4(at, f, first, make_float4(__uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])));
        }
    }
}

// The query tile.  A tile is read by one CTA only (by the few parts of a split one), so the rows come as the caller's f32 and become
// the two pieces here, between shared memory and the MMAs' operands: no planes of q are written and read again, and no
// launch before this one has to know q's maxima, so a small launch has its rows in place before the pre-pass ends.  Every row has
// a power of two of its own, which its thread takes out of the scores.  It costs a CTA about 1500 clocks before its first MMA (3500
// while a thread converted a row by itself).  Us, forward and backward, q's planes from the pre-pass -> rows: one sequence of 256, 4/2
// heads of 32 42.1 -> 39.1; batch 8, T 512, 32/8 heads of 64 255 -> 241; batch 4, T 1000, 16/4 of 80 248 -> 236; batch 8, T 1024, 32/8
// of 256 2580 -> 2410; T 4096, of 128 11970 -> 11640.
constexpr int kQBlock = 128 * 128;  // 32 columns of the tile's 128 rows, as TMA lands them: 128 bytes a row, swizzled
template <int D>
__device__ __forceinline__ void load_q(uint8_t *tile, const CUtensorMap *map, uint64_t *bar, int row, int head, int b) {
#pragma unroll
    for (int c = 0; c < D / 32; ++c) tma_load_4d(tile + c * kQBlock, map, bar, c * 32, head, row, b);
}
// Four columns of a row, whose bytes are its thread's alone.
__device__ __forceinline__ float4 *q_at(uint8_t *tile, int row, int chunk) {
    return reinterpret_cast<float4 *>(tile + (chunk >> 3) * kQBlock + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
}
// Rotates columns of the row in place: chunks [first, last) of the head's lower half (h4 chunks) and their partners, by the row's
// (cos, sin) pairs.
__device__ __forceinline__ void rotate_q(uint8_t *tile, int row, const float2 *angles, int h4, int first, int last) {
    for (int ch = first; ch < last; ++ch) {
        const float4 lo = *q_at(tile, row, ch), hi = *q_at(tile, row, h4 + ch);
        const float4 *cs = reinterpret_cast<const float4 *>(angles) + 2 * ch;
        float4 a, b;
        rope_chunk(lo, hi, cs[0], cs[1], a, b);
        *q_at(tile, row, ch) = a, *q_at(tile, row, h4 + ch) = b;
    }
}
__device__ __forceinline__ float max_abs4(float4 x) { return fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))); }
// The pieces of 32 columns times m: packed pairs of the hi ones, then of the lo ones.
template <class X>
__device__ __forceinline__ void split_q32(const X &column4, float m, uint32_t (&h)[16], uint32_t (&l)[16]) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float4 x = column4(c);
        split_pack(x.x * m, x.y * m, h[2 * c], l[2 * c]);
        split_pack(x.z * m, x.w * m, h[2 * c + 1], l[2 * c + 1]);
    }
}
// One piece each of the tile's 32 columns `block` into the K-major tile of halves that an MMA reads: half of a block of 64 columns.
__device__ __forceinline__ void store_q_piece(uint8_t *tile, int row, int block, const uint32_t (&l)[16]) {
    uint8_t *at = tile + (block >> 1) * kQBlock + row * 128;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        *reinterpret_cast<uint4 *>(at + ((((block & 1) * 4 + c) ^ (row & 7)) << 4)) = make_uint4(l[4 * c], l[4 * c + 1], l[4 * c + 2], l[4 * c + 3]);
}
// A finished row, or a part of it, from its thread's staging row in shared memory to `dst`, as one bulk copy: nothing of the warp waits
// for it but the end of the block.  (FLUSH: the row's running sum was written there by plain stores.)
template <bool FLUSH>
__device__ __forceinline__ void send_row(float *dst, const uint8_t *staged, int columns, bool wanted) {
    fence_async_smem();
    if (FLUSH) {  // (the sums of the warp's rows lie in each other's)
        asm volatile("fence.proxy.async.global;" ::: "memory");
        __syncwarp();
    }
    if (wanted && columns > 0) bulk_store(dst, staged, (uint32_t)columns * 4);
    tma_commit();
    tma_wait_read();
}

// A head's query row by two threads, which take a half of its columns each, out of their CTA's 256 (the barrier): hi pieces at TMEM `hi`,
// lo pieces at TMEM `lo` or, where LO_SMEM, over the tile (the rows have been read by then: a half goes where the row's columns
// of either thread were).  Returns the row's maximum; `tops` holds the halves'.
template <int D, bool LO_SMEM>
__device__ __forceinline__ float convert_q(uint8_t *tile, int set, int row, const float2 *angles, int dim, float (*tops)[128], uint32_t hi, uint32_t lo) {
    if (angles) {
        const int h4 = dim >> 3, mid = h4 >> 1;
        rotate_q(tile, row, angles, h4, set ? mid : 0, set ? h4 : mid);
        asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    float4 x[D / 8];
    float top = 0.f;
#pragma unroll
    for (int c = 0; c < D / 8; ++c) x[c] = *q_at(tile, row, set * (D / 8) + c), top = fmaxf(top, max_abs4(x[c]));
    tops[set][row] = top;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    top = fmaxf(top, tops[set ^ 1][row]);
    const float m = block_mult(__float_as_uint(top));
#pragma unroll
    for (int cb = 0; cb < D / 64; ++cb) {
        uint32_t qh[16], ql[16];
        split_q32([&](int c) { return x[cb * 8 + c]; }, m, qh, ql);
        tmem_st16(hi + set * (D / 4) + cb * 16, qh);
        if (LO_SMEM) store_q_piece(tile, row, set * (D / 64) + cb, ql);
        else tmem_st16(lo + set * (D / 4) + cb * 16, ql);
    }
    tmem_wait_st();
    if (LO_SMEM || angles) fence_async_smem();  // (what was written over the tile, before the copies that land there next)
    tc_fence_before();
    return top;
}
// The tile's maximum into its (sequence, KV group)'s, for the backward.
__device__ __forceinline__ void publish_q_top(const Params &p, int bg, float row_top) {
    if (p.amax_q == nullptr) return;
    const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(row_top));
    if ((threadIdx.x & 31) == 0) atomicMax(p.amax_q + bg, top);
}
// What turns a row's scores into log2 units, more than zero.  (One division after the other: a row of tiny values may have a scale
// whose product with k's is beyond f32.)
__device__ __forceinline__ float score_scale(float scale_log2, float mq, float mk) { return fmaxf(scale_log2 / mq / mk, 1.17549435e-38f); }

template <int D, bool FLUSH, bool PAD>
__global__ void __launch_bounds__(kThreads, 1)
    attn_fwd_tc16(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                  const __grid_constant__ CUtensorMap qmap, const Params p) {
    constexpr int NB = D / 64, W2 = D / 2, BN = 64;
    constexpr int KP = BN * D * 2;  // bytes of one plane of a key tile
    const bool padded = PAD && plane_dim(p.dim_out) < D;  // the planes are narrower than the tile
    constexpr int cQh = 0, cQl = W2, cO0 = D, cS0 = 3 * D;  // O of set s at cO0 + s D, S/P of buffer i at cS0 + 64 i
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *sK = smem, *sV = smem + 6 * KP;  // three slots of (hi, lo) each
    Shared *sh = reinterpret_cast<Shared *>(smem + 12 * KP);

    const int warp = threadIdx.x >> 5;
    // launch order (x fastest): a head's query tiles, late (long) ones first.  (Starting the heads of a sequence
    // tile by tile instead, which would shorten the tail, measured 3 % slower.)
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
        for (int i = 0; i < 3; ++i) {
            mbar_init(&sh->full_k[i], 1), mbar_init(&sh->free_k[i], 1);
            mbar_init(&sh->full_v[i], 1), mbar_init(&sh->free_v[i], 1);
        }
        mbar_init(&sh->a_ready, 8);
        for (int i = 0; i < 2; ++i) mbar_init(&sh->s_full[i], 1), mbar_init(&sh->p_full[i], 4), mbar_init(&sh->pv_done[i], 1);
        mbar_init(&sh->all_done, 1);
        mbar_init(&sh->q_full, 1);
        sh->abort = 0;
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
        // K of tile j is free again once S(j) has retired, two tiles before its V: rings of their own
        if (elect_one()) {
            tma_prefetch_desc(&qmap), tma_prefetch_desc(&kmap), tma_prefetch_desc(&vmap);
            // the query tile waits in V's first two slots until the row threads have its pieces in TMEM
            mbar_arrive_expect_tx(&sh->q_full, 4 * KP);
            load_q<D>(sV, &qmap, &sh->q_full, t0, h, b);
            pdl_wait();
            pdl_launch();
            int n_k = 0, n_v = 0;  // tiles issued
            bool live = true;
            const auto prefetch_next_q = [&]() {
                // The query tile of the CTA that will start when one of the running ones ends (`ahead` blocks on in
                // launch order, about the number of SMs), into L2: it would otherwise come from DRAM, under load, before
                // that CTA's first MMA can go out.
                const long long gx = gridDim.x, gy = gridDim.y;
                const long long lin = blockIdx.x + gx * (blockIdx.y + gy * blockIdx.z) + p.ahead;
                if (p.ahead <= 0 || lin >= gx * gy * gridDim.z) return;
                const int nx = (int)(lin % gx), ny = (int)((lin / gx) % gy), nz = (int)(lin / (gx * gy));
                const int nt0 = ((int)gx - 1 - nx) * 128;
                for (int c = 0; c < p.dim_out; c += 32) tma_prefetch_l2_4d(&qmap, c, ny, nt0, nz / p.parts);
            };
            auto load_k = [&](int j) {
                const int s = j % 3;
                if (j >= 3 && !fwait(&sh->free_k[s], (uint32_t)(((j / 3) & 1) ^ 1), sh)) { fgive_up(sh, 41), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_k[s], 2 * KP);
                load_head<NB>(sK + s * 2 * KP, &kmap, &sh->full_k[s], (jb + j) * BN, g, b, BN * 128, padded);
                load_head<NB>(sK + s * 2 * KP + KP, &kmap, &sh->full_k[s], (jb + j) * BN, g, B + b, BN * 128, padded);
                ++n_k;
            };
            auto load_v = [&](int j) {
                const int s = j % 3;
                if (j >= 3 && !fwait(&sh->free_v[s], (uint32_t)(((j / 3) & 1) ^ 1), sh)) { fgive_up(sh, 41), live = false; return; }
                mbar_arrive_expect_tx(&sh->full_v[s], 2 * KP);
                load_head<NB>(sV + s * 2 * KP, &vmap, &sh->full_v[s], (jb + j) * BN, g, b, BN * 128, padded);
                load_head<NB>(sV + s * 2 * KP + KP, &vmap, &sh->full_v[s], (jb + j) * BN, g, B + b, BN * 128, padded);
                ++n_v;
            };
            const int first = n_tiles < 3 ? n_tiles : 3;
            for (int j = 0; j < first; ++j) load_k(j);
            // V's slots are the query tile's until every row thread has its row in TMEM
            if (!fwait(&sh->a_ready, 0, sh)) fgive_up(sh, 41), live = false;
            for (int j = 0; live && j < first; ++j) load_v(j);
            prefetch_next_q();
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
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t id_s = idesc_f16(128, BN, false, false);
            const int steps = PAD ? head_steps(p.dim_out) : D / 16;
            const uint32_t id_o = idesc_f16(128, 16 * steps, false, true);
            bool ok = fwait(&sh->a_ready, 0, sh);
            if (!ok) fgive_up(sh, 42);
            tc_fence_after();
            const uint32_t k_u32 = smem_u32(sK), v_u32 = smem_u32(sV);
            // S of tile j into buffer j & 1
            auto issue_qk = [&](int j) -> bool {
                const int s = j % 3;
                if (!fwait(&sh->full_k[s], (uint32_t)((j / 3) & 1), sh)) return false;
                tc_fence_after();
                const uint32_t kh = k_u32 + (uint32_t)(s * 2 * KP);
                const uint64_t bkh = desc_kmajor(kh), bkl = desc_kmajor(kh + KP);
                const uint32_t cS = cS0 + (j & 1) * BN;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    if (PAD && kk >= steps) break;
                    const uint32_t bo = (uint32_t)((kk >> 2) * (BN * 128) + (kk & 3) * 32);
                    const uint64_t dkh = desc_advance(bkh, bo), dkl = desc_advance(bkl, bo);
                    mma_ts_f16(tmem + cS, tmem + cQh + kk * 8, dkh, id_s, kk > 0);
                    mma_ts_f16(tmem + cS, tmem + cQh + kk * 8, dkl, id_s, 1);
                    mma_ts_f16(tmem + cS, tmem + cQl + kk * 8, dkh, id_s, 1);
                }
                mma_commit(&sh->free_k[s]);
                mma_commit(&sh->s_full[j & 1]);
                return true;
            };
            if (ok && !issue_qk(0)) { fgive_up(sh, 43); ok = false; }
            if (ok && n_tiles > 1 && !issue_qk(1)) { fgive_up(sh, 43); ok = false; }
            for (int j = 0; ok && j < n_tiles; ++j) {
                const int s = j % 3, set = j & 1;
                if (!fwait(&sh->p_full[set], (uint32_t)((j >> 1) & 1), sh) ||
                    !fwait(&sh->full_v[s], (uint32_t)((j / 3) & 1), sh)) { fgive_up(sh, 44); break; }
                tc_fence_after();
                const uint32_t vh = v_u32 + (uint32_t)(s * 2 * KP);
                const uint64_t mvh = desc_mnmajor_16b(vh, BN * 128), mvl = desc_mnmajor_16b(vh + KP, BN * 128);
                const uint32_t cS = cS0 + set * BN, cO = cO0 + set * D;
                const bool fresh = j < 2 || (FLUSH && (j >> 1) % kFlushKeyTiles == 0);  // (O was flushed before tile j)
#pragma unroll
                for (int kk = 0; kk < BN / 16; ++kk) {
                    const uint32_t ac = (uint32_t)(32 * (kk >> 1) + (kk & 1) * 8);
                    const uint64_t dvh = desc_advance(mvh, kk * 2048), dvl = desc_advance(mvl, kk * 2048);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvh, id_o, (!fresh || kk > 0) ? 1 : 0);
                    mma_ts_f16(tmem + cO, tmem + cS + ac, dvl, id_o, 1);
                    mma_ts_f16(tmem + cO, tmem + cS + ac + 16, dvh, id_o, 1);
                }
                mma_commit(&sh->free_v[s]);
                mma_commit(&sh->pv_done[set]);
                // completes once, after the last P.V: a barrier that counts tiles may be two phases ahead
                // of a row thread by the time it gets there, which a parity wait cannot tell apart
                if (j == n_tiles - 1) mma_commit(&sh->all_done);
                // S(j+2) overwrites the P tile this P.V has just read
                if (j + 2 < n_tiles && !issue_qk(j + 2)) { fgive_up(sh, 43); break; }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ softmax rows: set `set` owns
        // the key tiles of its parity, with a reference maximum, a sum and an O accumulator of its own;
        // the two partial softmaxes are merged at the end.  Nothing a set does waits on the other's tile.
        const int tid = threadIdx.x & 127, set = threadIdx.x >> 7;
        const int t = t0 + tid, pos = p.q_offset + t;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        bool ok = true;
        float top;  // max |q| of the row
        {
            if (!__all_sync(0xffffffffu, fwait(&sh->q_full, 0, sh))) fgive_up(sh, 49), ok = false;
            const float2 *angles = p.rope ? p.rope + (long long)(t < p.T ? t : 0) * (p.dim_out >> 1) : nullptr;
            top = convert_q<D, false>(sV, set, tid, angles, p.dim_out, sh->q_top, tmem + lane_base + cQh, tmem + lane_base + cQl);
            mbar_arrive_warp(&sh->a_ready);
        }
        pdl_wait();
        const float mk = block_mult(p.amax_k[b * p.n_kv_heads + g]), mv = block_mult(p.amax_v[b * p.n_kv_heads + g]);
        if (set == 0) publish_q_top(p, b * p.n_kv_heads + g, top);
        const float cs = score_scale(p.scale_log2, block_mult(__float_as_uint(top)), mk);
        const uint32_t cS = cS0 + set * BN, cO = cO0 + set * D;
        float m_ref = -INFINITY, l = 0.f;
        float m_flushed = -INFINITY;  // the reference maximum of what has been flushed
        // where the sets keep flushed sums: set 0 in out, set 1 in rows of its own
        FlushRow row0{}, row1{};
        if (FLUSH) {
            float *rows = p.out + part * p.out_part;
            row0 = flush_row_at(p, rows, b, t0 + (warp & 3) * 32, h);
            row1 = flush_row_at(p, p.parts > 1 ? rows + p.parts * p.out_part : p.flush_rows, b, t0 + (warp & 3) * 32, h);  // (parts': behind the parts' rows)
        }
        for (int j = set; ok && j < n_tiles; j += 2) {
            if (!__all_sync(0xffffffffu, fwait(&sh->s_full[set], (uint32_t)((j >> 1) & 1), sh))) {
                fgive_up(sh, 45);
                ok = false;
                break;
            }
            tc_fence_after();
            const int s0 = (jb + j) * BN;
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
            const bool flush = FLUSH && j > 1 && (j >> 1) % kFlushKeyTiles == 0;
            const bool moved = __any_sync(0xffffffffu, factor != 1.f);
            if (j > 1 && (flush || moved)) {
                // this set's O may only be touched once its previous P.V (tile j-2) has retired
                if (!__all_sync(0xffffffffu, fwait(&sh->pv_done[set], (uint32_t)(((j >> 1) - 1) & 1), sh))) {
                    fgive_up(sh, 46);
                    ok = false;
                    break;
                }
                tc_fence_after();
                if (flush) {
                    const bool first = m_flushed == -INFINITY;
                    flush_row<D>(tmem + lane_base + cO, set == 0 ? row0 : row1, first ? 0.f : ex2(m_flushed - m_old), first);
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
        // ---- merge the two partial softmaxes
        sh->fin_m[set][tid] = m_ref;
        sh->fin_l[set][tid] = l;
        sh->fin_f[set][tid] = m_flushed;
        if (FLUSH) asm volatile("fence.proxy.async.global;" ::: "memory");  // (each set sends columns of the row that the other has summed, too)
        asm volatile("bar.sync 1, 256;" ::: "memory");  // the 256 softmax threads
        if (ok && !__all_sync(0xffffffffu, fwait(&sh->all_done, 0, sh))) {
            fgive_up(sh, 48);
            ok = false;
        }
        // The merged rows go to global memory through shared memory (K's slots: every tile has been consumed once all_done
        // completes), a half row of each thread as one bulk copy.  A row that goes to more places than out goes by stores, a row
        // (or two) an instruction.
        constexpr int RS = D * 4 + 16;  // (eight threads' chunks lie in different banks)
        const bool plain = p.o_planes == nullptr && p.out_peers.n == 0;
        uint8_t *srow = sK + tid * RS;
        if (ok) {
            tc_fence_after();
            const bool two = n_tiles > 1;  // set 1 has an accumulator only then
            const float m0 = sh->fin_m[0][tid], l0 = sh->fin_l[0][tid];
            const float m1 = two ? sh->fin_m[1][tid] : -INFINITY, l1 = two ? sh->fin_l[1][tid] : 0.f;
            // (finite where the CTA has all the keys, key 0 being visible to every row; a part may hold none that a row sees)
            const float mm = fmaxf(fmaxf(m0, m1), -3.0e38f);
            // (the merge is a running-maximum correction too, the only one where each set has a single tile)
            const float w0 = ZT_DEFECT(3) ? 1.f : ex2(m0 - mm), w1 = (m1 == -INFINITY) ? 0.f : (ZT_DEFECT(3) ? 1.f : ex2(m1 - mm));
            const float lsum = w0 * l0 + w1 * l1;
            const float inv = lsum == 0.f ? 0.f : 1.f / (lsum * mv);  // lsum, like O, carries kPScale
            const float f0 = w0 * inv, f1 = w1 * inv;
            const float s0 = sh->fin_f[0][tid], s1 = sh->fin_f[1][tid];
            const bool add0 = FLUSH && s0 != -INFINITY && row0.sums != nullptr, add1 = FLUSH && s1 != -INFINITY && row1.sums != nullptr;
            const float g0 = add0 ? ex2(s0 - m0) : 0.f, g1 = add1 ? ex2(s1 - m1) : 0.f;
            // set s merges columns [s D/2, (s+1) D/2) of the row
#pragma unroll 1
            for (int c = 0; c < D / 2; c += 32) {
                uint32_t ra[32], rb[32];
                tmem_ld32(tmem + lane_base + cO0 + set * (D / 2) + c, ra);
                if (two) tmem_ld32(tmem + lane_base + cO0 + D + set * (D / 2) + c, rb);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const int col = set * (D / 2) + c + i;
                    float4 o4 = make_float4(__uint_as_float(ra[i]), __uint_as_float(ra[i + 1]), __uint_as_float(ra[i + 2]), __uint_as_float(ra[i + 3]));
                    if (add0 && col < row0.width) o4 = flush_sum4(row0.at(col), g0, false, o4);
                    o4.x *= f0, o4.y *= f0, o4.z *= f0, o4.w *= f0;
                    if (two && w1 != 0.f) {
                        float4 x4 = make_float4(__uint_as_float(rb[i]), __uint_as_float(rb[i + 1]), __uint_as_float(rb[i + 2]), __uint_as_float(rb[i + 3]));
                        if (add1 && col < row1.width) x4 = flush_sum4(row1.at(col), g1, false, x4);
                        o4.x += x4.x * f1, o4.y += x4.y * f1, o4.z += x4.z * f1, o4.w += x4.w * f1;
                    }
                    *reinterpret_cast<float4 *>(srow + col * 4) = o4;
                }
            }
            if (set == 0 && p.lse && t < p.T)
                p.lse[part * p.lse_part + ((long long)b * p.T + t) * p.n_heads + h] = (mm + log2f(lsum) - 7.0f) * kLn2;
        }
        if (FLUSH) asm volatile("bar.sync 1, 256;" ::: "memory");  // (either set has read sums out of the rows that the other sends to)
        if (plain) {
            const int c0 = set * (D / 2), mine = p.dim_out - c0 < D / 2 ? p.dim_out - c0 : D / 2;
            send_row<FLUSH>(p.out + part * p.out_part + (((long long)b * p.T + t) * p.n_heads + h) * p.dim_out + c0, srow + c0 * 4, mine, ok && t < p.T);
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (!plain && !sh->abort) {
            constexpr int CH = D / 4;  // 16-byte chunks per row
            constexpr int RPI = 32 / CH;  // rows per store instruction
            const int lane = threadIdx.x & 31;
            const int ch = lane & (CH - 1);
            const long long wo = (long long)p.n_heads * p.dim_out;
            const float mo = p.o_planes ? out_plane_mult(p, b) : 1.f;
#pragma unroll 4
            for (int i = 0; i < 16; i += RPI) {
                const int r = warp * 16 + i + lane / CH;
                const float4 o4 = *reinterpret_cast<const float4 *>(sK + r * RS + ch * 16);
                if (t0 + r < p.T && ch * 4 < p.dim_out)  // (a padded tile's upper columns are not the tensor's)
                    store_out4(p, part * p.out_part + ((long long)b * p.T + t0 + r) * wo + (long long)h * p.dim_out + ch * 4, o4, mo);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem, 512);
}


struct Workspace {
    uint32_t *amax_q, *amax_k, *amax_v;
    uint32_t *vnmax;  // (in the backward's layout: the largest row norm of v, which the backward wants; else null)
    uint2 *part[3];   // the pre-pass's slots
    float *flush_rows;  // (see Params)
    __half *k_planes, *v_planes;
    float *parts;     // of a forward split along the keys: behind everything else
    size_t base_bytes, total_bytes;
};

inline Workspace workspace(void *base, int batch, int T, int n_heads, int n_kv_heads, int dim, int q_offset = 0) {
    Workspace w{};
    const size_t n_amax = (size_t)batch * n_kv_heads;
    auto up = [](size_t x) { return (x + 1023) / 1024 * 1024; };
    const size_t rows = (size_t)batch * T * n_heads * dim * sizeof(float);
    const size_t kh = (size_t)2 * batch * (q_offset + T) * n_kv_heads * dim * sizeof(__half);
    char *c = static_cast<char *>(base);
    w.amax_q = reinterpret_cast<uint32_t *>(c), w.amax_k = w.amax_q + n_amax, w.amax_v = w.amax_k + n_amax;
    size_t off = up(3 * n_amax * sizeof(uint32_t));
    for (int i = 0; i < 3; ++i) w.part[i] = reinterpret_cast<uint2 *>(c + off), off += up(tcb::pass_part_bytes(n_amax));
    w.flush_rows = reinterpret_cast<float *>(c + off), off += up(rows);
    w.k_planes = reinterpret_cast<__half *>(c + off), off += up(kh);
    w.v_planes = reinterpret_cast<__half *>(c + off), off += up(kh);
    w.base_bytes = off;
    w.parts = reinterpret_cast<float *>(c + off), off += up(fwd_parts_floats(batch, T, n_heads, dim, q_offset) * sizeof(float));
    w.total_bytes = off;
    return w;
}

template <int D>
inline int launch_d(const CUtensorMap &kmap, const CUtensorMap &vmap, const CUtensorMap &qmap, const Params &p,
                    cudaStream_t stream) {
    size_t smem = 12 * (size_t)(64 * D * 2) + sizeof(Shared) + 1024;
    if (smem < 120 * 1024) smem = 120 * 1024;  // one CTA per SM: it allocates all of TMEM
    const auto kernel = with_flags([](auto flush, auto pad) { return attn_fwd_tc16<D, flush.value, pad.value>; }, p.flush, head_steps(p.dim_out) < D / 16);
    if (optin_smem((const void *)kernel, smem)) return 1;
    const dim3 grid = p.by_tile ? tile_major_grid(p.n_heads, (p.T + 127) / 128, p.batch * p.parts, kFwdTileWaves)
                                : dim3((unsigned)((p.T + 127) / 128), (unsigned)p.n_heads, (unsigned)(p.batch * p.parts));
    return launch_after("attn_fwd_tc16", kernel, grid, dim3(kThreads), smem, stream, 1, kmap, vmap, qmap, p);
}

// (tc_fwd16x.cuh)
template <int D>
inline int launch_x_d(const CUtensorMap &kmap, const CUtensorMap &vmap, const CUtensorMap &qmap, const Params &p,
                    cudaStream_t stream);
// (tc_fwd16g.cuh)
template <int D>
inline int launch_g_d(const CUtensorMap &kmap, const CUtensorMap &vmap, const CUtensorMap &qmap, const Params &p,
                      cudaStream_t stream);
// (tc_fwd16n.cuh)
inline int launch_n(const CUtensorMap &kmap, const CUtensorMap &vmap, const CUtensorMap &qmap, Params p, int sms, cudaStream_t stream);

}  // namespace tcf16

inline size_t tc_fwd16_workspace_bytes(int batch, int T, int n_heads, int n_kv_heads, int dim, int q_offset = 0) {
    return tcf16::workspace(nullptr, batch, T, n_heads, n_kv_heads, tc::plane_dim(dim), q_offset).total_bytes;
}

inline bool tc_fwd16_supported(int batch, int T, int q_offset, int dim, const void *q, const void *k, const void *v, const void *out) {
    if (!tc_takes_dim(dim) || q_offset + T < kTcForwardMinKeys || batch < 1) return false;
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (!al(q) || !al(k) || !al(v) || !al(out)) return false;
    const DeviceInfo *d = device_info();
    return d && d->cc_major == 10 && get_encode_tiled() != nullptr;
}

// `in_backward_workspace`: lay the planes out where the backward's workspace keeps them (tc_bwd.cuh
// bwd_workspace), so that a backward given the same workspace can use them as they are.
// q_offset: the query rows are a window of the sequence that starts there (batch 1; k and v hold at least q_offset + T
// rows, of which the later ones are not read).
// out_planes (optional): where the kernel also leaves out as f16 hi/lo planes, [2][batch][T][n_heads * dim] halves.
// ws_bytes: at least the layout's bytes without the parts; a forward that has no room for them is not split.
inline int launch_fwd_tc16(const float *q, const float *k, const float *v, float *out, float *lse, void *ws, size_t ws_bytes,
                           int batch, int T, int n_heads, int n_kv_heads, int dim, cudaStream_t stream,
                           const float2 *rope = nullptr, bool in_backward_workspace = false, int variant = 0,
                           __half *out_planes = nullptr, const PeerList *out_peers = nullptr, int q_offset = 0) {
    using namespace tcb;
    const int td = tc_tile_dim(dim), pd = tc::plane_dim(dim);  // the kernel's D; the planes' head width
    tcf16::Workspace w = tcf16::workspace(ws, batch, T, n_heads, n_kv_heads, pd, q_offset);
    if (in_backward_workspace) {
        const BwdWorkspace bw = bwd_workspace(ws, batch, T, n_heads, n_kv_heads, pd);
        w.amax_q = bw.amax_q, w.amax_k = bw.amax_k, w.amax_v = bw.amax_v;
        w.vnmax = bw.vnmax;
        for (int i = 0; i < 3; ++i) w.part[i] = bw.part[i];
        w.k_planes = bw.k_planes, w.v_planes = bw.v_planes, w.parts = bw.parts;
        w.base_bytes = bw.base_bytes;
    }
    const int group = n_heads / n_kv_heads;
    const int n_seen = q_offset + T;  // key rows that some query row sees
    PassArgs pa{};
    pa.dim = dim, pa.pd = pd, pa.q_units = T * group;
    {
        PassTensor &t = pass_add(pa, k, batch, n_seen, n_kv_heads, 1, w.part[1], w.amax_k, nullptr, w.k_planes);
        t.rope = rope;
        if (in_backward_workspace) t.clear = w.amax_q;
    }
    pass_add(pa, v, batch, n_seen, n_kv_heads, 1, w.part[2], w.amax_v, w.vnmax, w.v_planes);
    if (launch_pass(pa, stream)) return 1;
    CUtensorMap kmap, vmap, qmap;  // (the widest tiles fetch K block by block and V by 16 keys, see attn_fwd_tc16x)
    if (!make_head_map(&kmap, w.k_planes, 2 * batch, n_seen, n_kv_heads, dim, td > 128 ? 1 : td / 64, 64) ||
        !make_head_map(&vmap, w.v_planes, 2 * batch, n_seen, n_kv_heads, dim, td / 64, td > 128 ? 16 : 64) ||
        !make_row_map(&qmap, q, batch, T, n_heads, dim, 128))
        return refuse("the TMA tensor maps for the forward could not be encoded.");
    const int sms = split_sm_count();
    tcf16::Params p{};
    p.amax_q = in_backward_workspace ? w.amax_q : nullptr, p.amax_k = w.amax_k, p.amax_v = w.amax_v;
    p.rope = rope, p.flush_rows = q_offset > 0 ? w.flush_rows : nullptr;
    p.out = out, p.lse = lse;
    p.batch = batch, p.T = T, p.n_heads = n_heads, p.n_kv_heads = n_kv_heads;
    p.dim_out = dim, p.q_offset = q_offset;
    p.o_planes = out_planes, p.o_plane_stride = (long long)batch * T * n_heads * dim;
    if (out_peers) p.out_peers = *out_peers;
    p.scale_log2 = kLog2e / sqrtf((float)dim);
    p.parts = variant == 0 && !out_planes && p.out_peers.n == 0 ? fwd_parts(batch, T, n_heads, q_offset) : 1;
    if (p.parts > 1 && w.base_bytes + fwd_parts_floats(batch, T, n_heads, pd, q_offset) * sizeof(float) > ws_bytes) p.parts = 1;
    const long long rows = (long long)batch * T * n_heads;
    if (p.parts > 1) {
        p.out = w.parts, p.out_part = rows * dim;
        p.lse = w.parts + p.parts * (q_offset > 0 ? 2 : 1) * p.out_part, p.lse_part = rows;
    }
    p.by_tile = tile_by_tile((long long)((T + 127) / 128) * n_heads * batch * p.parts, kFwdTileWaves);
    p.ahead = p.by_tile ? 0 : sms;  // one CTA per SM
    g_last_path = "tcgen05";
    // variant 0: two heads of a KV group per CTA (attn_fwd_tc16g) when the group has an even number of query heads
    // and that still gives every SM a CTA (half as many CTAs), one head per CTA (attn_fwd_tc16) otherwise; 1: one head
    // per CTA; 2: two heads per CTA whatever the number of CTAs (the group must be even).
    const long long pair_ctas = (long long)((T + 127) / 128) * (n_heads / 2) * batch;
    const bool pairs = td <= 128 && group % 2 == 0 && (variant == 2 || (variant == 0 && pair_ctas >= sms));
    const long long blocks = (long long)((T + 127) / 128) * n_heads * batch;
    // Up to 64 columns, with more than a CTA an SM: two an SM (attn_fwd_tc16n).  Below, one tile at a time, two softmax sets in turn are the
    // quicker; and up to two CTAs an SM, whose launch ends with its longest walk, for long sequences too.  Us, one head a CTA / two CTAs an
    // SM: 160 CTAs, T 1000 26.4 / 23.8, 2000 192 CTAs 36.8 / 39.4, 3000 192 46.1 / 51.9, 288 53.6 / 57.3, 4500 288 75.6 / 91.1, 7000 220
    // 91 / 123; T 1400 176 30.2 / 30.4, 264 36.5 / 33.7; T 700 288 30.8 / 23.2.  (A window's walks are all of a length: 1400 rows at 3000
    // keys, 176 CTAs, 112.8 / 112.6.)  Windows of fewer than two waves of pairs stay with two heads a CTA: neither is the quicker throughout.
    // Us, two heads a CTA / two CTAs an SM: 1200 rows at 1100 keys, 32/8 heads of 64 85 / 78, 1500 at 2500, of 56 162 / 155, 1300 at
    // 6000 309 / 304, 4000 at 4000, 16/4 287 / 306, 2200 at 9000, 32/8 503 / 531.  (The shortest lose by it; a test holds 1200 at 1100 there.)
    const bool narrow = td == 64 && variant == 0 && p.parts == 1 && blocks > sms && !(q_offset == 0 && blocks < 2LL * sms && T > 1536) &&
                        !(q_offset > 0 && pairs && pair_ctas < 2LL * sms);
    // An accumulator that takes no more than kFlushKeyTiles tiles is never flushed: the variant without, whose end has no sums to look for.  (A CTA of one head
    // gives its tiles to two accumulators in turn up to 128 columns.)  Us, 100 rows at 1700 keys, 12/4 heads of 96 20.2 -> 19.6, 200 at 3000 29.9 -> 29.0.
    const int tiles = (n_seen + 63) / 64, per = (tiles + p.parts - 1) / p.parts;
    p.flush = q_offset > 0 && per > tcf16::kFlushKeyTiles * (td <= 128 && (narrow || !pairs) ? 2 : 1);
    int rc;
    if (narrow) rc = tcf16::launch_n(kmap, vmap, qmap, p, sms, stream);
    else if (td == 256) rc = tcf16::launch_x_d<256>(kmap, vmap, qmap, p, stream);
    else if (td == 192) rc = tcf16::launch_x_d<192>(kmap, vmap, qmap, p, stream);
    else if (pairs) rc = td == 64 ? tcf16::launch_g_d<64>(kmap, vmap, qmap, p, stream) : tcf16::launch_g_d<128>(kmap, vmap, qmap, p, stream);
    else rc = td == 64 ? tcf16::launch_d<64>(kmap, vmap, qmap, p, stream) : tcf16::launch_d<128>(kmap, vmap, qmap, p, stream);
    if (rc || p.parts == 1) return rc;
    return launch_fwd_join(p.out, p.lse, out, lse, rows, dim, p.parts, stream);
}

}  // namespace zt
