// Causal GQA attention forward of up to 128 keys on tiles of 64 and 128 columns, in one launch.
//
// The other tensor-core forwards read f16 operand planes that two launches before them leave in memory: one for the largest
// magnitude of every (sequence, KV group), which sets the planes' scale, and one for the planes.  A short prompt is nothing but
// the latency of that chain.  Here a block has one head's whole q, k and v in registers (a tile of 128 rows each), so that it
// knows their maxima after one barrier, splits them itself and leaves the operands in shared memory as TMA would have:
//   S = Qh.Kh + Qh.Kl + Ql.Kh      one accumulator of 128 x (keys, up to a multiple of 16)
//   P = exp(S - max) 2^7           four warps a 32-column quarter of S, a row's maximum and sum put together through shared memory
//   O = Pl.Vh + Ph.Vl + Ph.Vh      P in TMEM over S, V read N-major
// with the arithmetic of attn_fwd_tc16 (three-term split on f16 pieces, f32 accumulators).  S's terms are added in its order, which is
// the backwards' too: the tensor core truncates, and a backward that adds S otherwise than the forward whose out and log-sum-exp it
// is given finds another P (T 128, scores that rise with the key, dq against float64, small terms first -> so: heads of 32 2.8e-6 ->
// 1.1e-6, of 128 2.3e-6 -> 1.7e-6).  O's small terms go first, while there is little to truncate.
// Every query head converts its KV head's k and v again; a group's heads run side by side, and even several waves of blocks, each
// of which does so, are faster than the planes' two launches: us, planes -> this, one prompt of 77, 32/8 heads of 128 17.0 -> 8.3, of 40,
// 4/2 of 32 12.9 -> 5.1; 8 prompts of 100, 32/8 of 128 42 -> 21, 16 of 128 70 -> 46; 16 of 128, 32/8 of 64 43 -> 29.
// What bounds it: latency, in this order -- the launch, q, k and v from memory, the two chains of MMAs, the rows' way out.
#pragma once

#include "tc_fwd16.cuh"

namespace zt {
namespace tcshort {

using namespace tc;
using tcb::block_mult;
using tcb::split_pack;

constexpr int kMaxKeys = 128, kThreads = 512;

struct Shared {
    uint64_t s_full, o_full;
    uint32_t tmem_base;
    volatile int abort;
    uint32_t top[3][kThreads / 32];   // each warp's largest |q|, |k|, |v|
    float m[4][128], l[4][128];       // each quarter's maximum and sum of every row
};
struct Params {
    const float *q, *k, *v;
    float *out, *lse;                 // lse may be null
    int T, q_offset, n_heads, n_kv_heads, dim;
    long long kv_batch;               // elements from one sequence's k or v to the next
    float scale_log2;
};
__device__ __forceinline__ bool swait(uint64_t *bar, Shared *sh) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        if (mbar_try_wait(bar, 0)) return true;
        if ((i & 255u) == 255u && sh->abort) return false;
    }
    return false;
}

// grid (n_heads, batch), 512 threads
template <int D>
__global__ void __launch_bounds__(kThreads, 1) attn_fwd_short(const Params p) {
    constexpr int LP = D / 4, R = kThreads / LP, NP = 128 / R;  // lanes a row, rows a pass, passes over a tile
    constexpr int BT = 128 * 128, PB = D / 64 * BT;             // bytes of a 64-column block of 128 rows; of an operand plane
    constexpr int cS = 0, cO = 128;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *sQ = smem, *sK = smem + 2 * PB, *sV = smem + 4 * PB;  // hi, lo each
    Shared *sh = reinterpret_cast<Shared *>(smem + 6 * PB);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.x, b = blockIdx.y, g = h / (p.n_heads / p.n_kv_heads);
    const int n_keys = p.q_offset + p.T, kn = (n_keys + 15) & ~15;
    const int li = threadIdx.x % LP, ri = threadIdx.x / LP;
    const bool in = li * 4 < p.dim;

    pdl_wait();
    float4 x[3][NP];
    {
        const float *q = p.q + ((long long)b * p.T * p.n_heads + h) * p.dim + li * 4;
        const long long kv0 = b * p.kv_batch + (long long)g * p.dim + li * 4;
        const int wq = p.n_heads * p.dim, wkv = p.n_kv_heads * p.dim;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const int r = i * R + ri;
            x[0][i] = in && r < p.T ? *reinterpret_cast<const float4 *>(q + (long long)r * wq) : zero;
            x[1][i] = in && r < n_keys ? *reinterpret_cast<const float4 *>(p.k + kv0 + (long long)r * wkv) : zero;
            x[2][i] = in && r < n_keys ? *reinterpret_cast<const float4 *>(p.v + kv0 + (long long)r * wkv) : zero;
        }
    }
    // (set up while the loads are on their way)
    if (threadIdx.x == 0) {
        mbar_init(&sh->s_full, 1), mbar_init(&sh->o_full, 1);
        sh->abort = (smem_u32(smem) & 1023u) ? 30 : 0;
        if (sh->abort) atomicMax(&g_tc_status, 30);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&sh->tmem_base, 256);
#pragma unroll
    for (int z = 0; z < 3; ++z) {
        float top = 0.f;
#pragma unroll
        for (int i = 0; i < NP; ++i)
            top = fmaxf(top, fmaxf(fmaxf(fabsf(x[z][i].x), fabsf(x[z][i].y)), fmaxf(fabsf(x[z][i].z), fabsf(x[z][i].w))));
        const uint32_t t = __reduce_max_sync(0xffffffffu, __float_as_uint(top));  // (bit patterns of non-negative numbers order like integers)
        if (lane == 0) sh->top[z][warp] = t;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch();  // (only now that the block has its TMEM: a successor that took more of it ahead of its own pdl_wait would wait for this grid)
    const uint32_t tmem = sh->tmem_base;
    float mult[3];
#pragma unroll
    for (int z = 0; z < 3; ++z) {
        const uint32_t t = __reduce_max_sync(0xffffffffu, sh->top[z][lane & (kThreads / 32 - 1)]);
        mult[z] = block_mult(t);
        // rows of 128 bytes, 128-byte swizzled: what a TMA copy of the planes' tile leaves
        uint8_t *hi = smem + z * 2 * PB + (li >> 4) * BT + (li & 1) * 8;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const int r = i * R + ri;
            if (r >= (z == 0 ? p.T : kn)) break;  // (a query row past the tensor's leaves what is there: it reaches no other row)
            uint2 hw, lw;
            split_pack(x[z][i].x * mult[z], x[z][i].y * mult[z], hw.x, lw.x);
            split_pack(x[z][i].z * mult[z], x[z][i].w * mult[z], hw.y, lw.y);
            const int at = r * 128 + ((((li & 15) >> 1) ^ (r & 7)) << 4);
            *reinterpret_cast<uint2 *>(hi + at) = hw;
            *reinterpret_cast<uint2 *>(hi + PB + at) = lw;
        }
    }
    fence_async_smem();
    __syncthreads();
    const int steps = head_steps(p.dim), key_steps = kn / 16;
    if (warp == 0) {
        if (elect_one() && !sh->abort) {
            const uint32_t id_s = idesc_f16(128, kn, false, false);
            const uint64_t qh = desc_kmajor(smem_u32(sQ)), ql = desc_kmajor(smem_u32(sQ) + PB);
            const uint64_t kh = desc_kmajor(smem_u32(sK)), kl = desc_kmajor(smem_u32(sK) + PB);
#pragma unroll 1
            for (int kk = 0; kk < steps; ++kk) {
                const uint32_t o = (uint32_t)((kk >> 2) * BT + (kk & 3) * 32);
                mma_ss_f16(tmem + cS, desc_advance(qh, o), desc_advance(kh, o), id_s, kk > 0);
                mma_ss_f16(tmem + cS, desc_advance(qh, o), desc_advance(kl, o), id_s, 1);
                mma_ss_f16(tmem + cS, desc_advance(ql, o), desc_advance(kh, o), id_s, 1);
            }
            mma_commit(&sh->s_full);
        }
        __syncwarp();
    }
    bool ok = __all_sync(0xffffffffu, swait(&sh->s_full, sh));
    if (!ok) sh->abort = 31, atomicMax(&g_tc_status, 31);
    tc_fence_after();
    // a thread per row and 32 of its keys
    const int row = (warp & 3) * 32 + lane, quarter = warp >> 2, key0 = quarter * 32, pos = ZT_DEFECT(1) ? n_keys - 1 : p.q_offset + row;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const bool some = key0 < kn;
    const float cs = tcf16::score_scale(p.scale_log2, mult[0], mult[1]);
    uint32_t r[32];
    float m = -INFINITY;
    if (some) {
        tmem_ld32(tmem + lane_base + cS + key0, r);
        tmem_wait_ld();
        tcf16::mask32(r, pos - key0);
        m = tcf16::row_max32(r, m) * cs;
    }
    sh->m[quarter][row] = m;
    __syncthreads();
    const float top = fmaxf(fmaxf(sh->m[0][row], sh->m[1][row]), fmaxf(sh->m[2][row], sh->m[3][row]));
    if (!ZT_DEFECT(3)) m = top;
    const float off = (m == -INFINITY ? 0.f : m) - 7.0f;  // log2 kPScale
    float sum = 0.f;
    if (some) {
        uint32_t ph[16], pl[16];
        sum = tcf16::row_exp32(r, cs, off, ph, pl);
        tmem_st16(tmem + lane_base + cS + key0, ph);
        tmem_st16(tmem + lane_base + cS + key0 + 16, pl);
        tmem_wait_st();
    }
    sh->l[quarter][row] = sum;
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        if (elect_one() && !sh->abort) {
            tc_fence_after();
            const uint32_t id_o = idesc_f16(128, 16 * steps, false, true);
            const uint64_t vh = desc_mnmajor_16b(smem_u32(sV), BT), vl = desc_mnmajor_16b(smem_u32(sV) + PB, BT);
#pragma unroll 1
            for (int kk = 0; kk < key_steps; ++kk) {
                const uint32_t a = tmem + cS + (kk >> 1) * 32 + (kk & 1) * 8;  // (32 keys: 16 columns of hi pairs, then their lo pairs)
                const uint64_t dvh = desc_advance(vh, kk * 2048), dvl = desc_advance(vl, kk * 2048);
                mma_ts_f16(tmem + cO, a, dvl, id_o, kk > 0);
                mma_ts_f16(tmem + cO, a + 16, dvh, id_o, 1);
                mma_ts_f16(tmem + cO, a, dvh, id_o, 1);
            }
            mma_commit(&sh->o_full);
        }
        __syncwarp();
    }
    const float l = (sh->l[0][row] + sh->l[1][row]) + (sh->l[2][row] + sh->l[3][row]);
    ok = __all_sync(0xffffffffu, swait(&sh->o_full, sh)) && ok;
    if (!ok) sh->abort = 32, atomicMax(&g_tc_status, 32);
    tc_fence_after();
    // the rows leave through shared memory (Q's, which has been read), whole rows at a time
    const float inv = l == 0.f ? 0.f : 1.f / (l * mult[2]);  // (l, like O, carries kPScale)
    {
        constexpr int Q4 = D / 4;  // a quarter's columns
        uint32_t o[Q4];
        if constexpr (Q4 == 32) tmem_ld32(tmem + lane_base + cO + quarter * Q4, o);
        else tmem_ld16(tmem + lane_base + cO + quarter * Q4, o);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < Q4; i += 4) {
            const int c = quarter * (Q4 / 4) + i / 4;
            *reinterpret_cast<float4 *>(sQ + row * (D * 4) + ((c ^ (row & (LP - 1))) << 4)) =
                make_float4(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv, __uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
        }
    }
    if (quarter == 0 && p.lse && ok && row < p.T) p.lse[((long long)b * p.T + row) * p.n_heads + h] = (top + log2f(l) - 7.0f) * kLn2;
    tc_fence_before();
    __syncthreads();
    if (ok && in) {
        float *out = p.out + ((long long)b * p.T * p.n_heads + h) * p.dim + li * 4;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const int t = i * R + ri;
            if (t >= p.T) break;
            *reinterpret_cast<float4 *>(out + (long long)t * p.n_heads * p.dim) = *reinterpret_cast<const float4 *>(sQ + t * (D * 4) + ((li ^ (t & (LP - 1))) << 4));
        }
    }
    if (warp == 1) tmem_dealloc(tmem, 256);
}

template <int D>
inline int launch_d(const Params &p, int batch, cudaStream_t stream) {
    const size_t smem = (size_t)6 * (D / 64) * 128 * 128 + sizeof(Shared);
    if (optin_smem((const void *)attn_fwd_short<D>, smem)) return 1;
    return launch_after("attn_fwd_short", attn_fwd_short<D>, dim3((unsigned)p.n_heads, (unsigned)batch), dim3(kThreads), smem, stream, 1, p);
}

}  // namespace tcshort

// Which forwards take it: every key in one tile, heads of up to 128 columns, for any number of blocks.  At its far end every one of a group's
// query heads converts the same k and v again: us, planes -> this, T 33, heads of 32, batch 2048, 32/8 heads 1978 -> 1950, 32/2 1938 -> 1907,
// 32/1 1844 -> 1897; 64/1, batch 128 234 -> 227, 256 467 -> 479, 1024 1811 -> 1896; 64/1 heads of 48 1962 -> 1952; T 100, 64/1 of 32, batch
// 256 649 -> 637.  (What 32 query heads a group lose beyond 8192 blocks is not worth a scratch, which leaves memory nodes in a graph.)
inline bool tc_fwd_short_takes(int batch, int T, int q_offset, int dim) {
    return q_offset + T <= tcshort::kMaxKeys && dim <= 128 && batch <= 65535;
}

// (after tc_fwd16_supported)  k and v hold n_keys rows a sequence, of which those from q_offset + T on are not read.
inline int launch_fwd_short(const float *q, const float *k, const float *v, float *out, float *lse, int batch, int T, int q_offset, int n_keys,
                            int n_heads, int n_kv_heads, int dim, cudaStream_t stream) {
    tcshort::Params p{};
    p.q = q, p.k = k, p.v = v, p.out = out, p.lse = lse;
    p.T = T, p.q_offset = q_offset, p.n_heads = n_heads, p.n_kv_heads = n_kv_heads, p.dim = dim;
    p.kv_batch = (long long)n_keys * n_kv_heads * dim;
    p.scale_log2 = kLog2e / sqrtf((float)dim);
    g_last_path = "tcgen05";
    return dim <= 64 ? tcshort::launch_d<64>(p, batch, stream) : tcshort::launch_d<128>(p, batch, stream);
}

}  // namespace zt
