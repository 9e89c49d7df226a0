// KV-cache decode attention: one new query row per sequence over that sequence's
// filled cache prefix (decode.attnStep, src/decode.zig:326-392, for a whole batch).
//
// The work is a stream over the cache -- every K and V row of every KV head is
// read exactly once and used by all query heads of its group -- so the kernel is
// bound by HBM bandwidth and everything here is arranged around that:
//   * split-K over the context: block (chunk, kv head, sequence) reads a fixed-size
//     chunk of keys, so ragged lengths balance by themselves and a short batch
//     still fills the machine;
//   * a K/V row is read by a group of LPK lanes as 128-bit, fully coalesced asynchronous
//     copies into shared memory, several steps ahead of their use;
//   * a row is read once and dotted against every query head of the group held
//     in registers; lane-group shuffles finish each dot;
//   * online softmax in the log2 domain per lane group, merged across lane
//     groups by shuffles, across warps through shared memory, and across the blocks of
//     a sequence's KV head either inside a thread-block cluster (its blocks divide the
//     keys evenly and read each other's sums from shared memory: one launch, nothing
//     in global memory) or, for contexts too long for that, by a second small
//     kernel over partial results in the workspace (log-sum-exp combine).
//
// Algorithmic bytes per sequence step: n_keys * 2 * n_kv_heads * dim * 4 (K and V
// once each) plus q and out.
#pragma once

#include "zt_common.cuh"

namespace zt {

constexpr int kDecodeThreads = 256;
constexpr int kMaxCluster = 8;
constexpr int kDecodeHeaderBytes = 256;  // workspace header: bad-sequence counter

struct DecodeParams {
    const float *q, *k_cache, *v_cache;
    const int *n_keys;  // per sequence; when null, n_keys_all applies to every sequence
    int n_keys_all;
    float *out, *lse;  // lse may be null
    float2 *part_ml;   // [batch, n_heads, max_chunks]  (running max (log2), denominator)
    float *part_acc;   // [batch, n_heads, max_chunks, dim]
    int *bad_count;    // in the workspace header
    int batch, n_ctx, n_heads, n_kv_heads, dim, chunk, max_chunks, n_sub;
    int cluster;  // blocks per cluster in the one-launch form
    long long cache_batch_stride;  // elements between two sequences' caches
    float scale_log2;
};

// How many sequences name no valid prefix: counted by one block, so that nothing has to be cleared beforehand.
__device__ __forceinline__ void count_bad_sequences(const DecodeParams &p) {
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    if (p.n_keys)
        for (int i = threadIdx.x; i < p.batch; i += blockDim.x)
            if (p.n_keys[i] < 1 || p.n_keys[i] > p.n_ctx) atomicAdd(&total, 1);
    __syncthreads();
    if (threadIdx.x == 0) *p.bad_count = total;
}

constexpr float kNoKey = -3.402823466e38f;  // the running maximum before the first key
constexpr float kDecodeLazy = 8.f;          // a maximum moves when it is outgrown by 2^8

// Blocks an SM holds, from a register estimate (q and accumulators: 8 floats per chunk per head).
__host__ __device__ constexpr int decode_blocks_per_sm(int nch, int gp) { return gp * nch * 8 + 56 > 128 ? 1 : 2; }

template <int LPK, int NCH, int GP>
struct DecodeCfg {
    // Keys a lane group takes per step: at most as many (key, head) pairs as it has lanes, and 128 bytes a thread.
    static constexpr int kUnroll = (4 / NCH < 1 ? 1 : 4 / NCH) * GP > LPK ? LPK / GP : (4 / NCH < 1 ? 1 : 4 / NCH);
    // Stages from what is left of shared memory (96 KB or 192 KB a block).
    static constexpr int kMinBlocks = decode_blocks_per_sm(NCH, GP);
    static constexpr int kStageBytes = kDecodeThreads * kUnroll * NCH * 2 * 16;
    static constexpr int kFit = (kMinBlocks == 2 ? 96 : 192) * 1024 / kStageBytes;
    static constexpr int kStages = kFit > 8 ? 8 : kFit;
};

// LPK lanes share one key row; each lane holds NCH float4 chunks of it (chunk index
// li + LPK * c); GP query heads are processed per pass.
// CLUSTER: the blocks of a cluster (x) divide the sequence's keys evenly and finish the rows among themselves;
// otherwise block x takes the x-th chunk of p.chunk keys and leaves a partial result.
//
// The loads run kStages - 1 steps ahead through slots of shared memory that belong to one thread each, filled by
// cp.async and waited for by that thread alone: no barrier in the loop, and the memory system always has 64 KB a block
// to work on.  (Held in registers, a step's loads could not go out before the step before had been used up: batch 64, 8192
// keys, 32/8 heads of 128 took 785 us, 5.5 TB/s; now 636 us, 6.75 TB/s.)
// The U GP dots of a step are summed over the lane group by exchanging halves -- V - 1 + log2(LPK / V) shuffles instead of
// V log2(LPK) -- which leaves each lane the sum of one (key, head) pair; that lane alone takes the exponential and keeps
// the head's maximum and its share of the denominator, and hands P out to the others.
template <int LPK, int NCH, int GP, bool CLUSTER>
__global__ void __launch_bounds__(kDecodeThreads, DecodeCfg<LPK, NCH, GP>::kMinBlocks)
    decode_splitk_kernel(const DecodeParams p) {
    using Cfg = DecodeCfg<LPK, NCH, GP>;
    constexpr int U = Cfg::kUnroll, S = Cfg::kStages;
    constexpr int V = U * GP, SP = LPK / V;                // (key, head) pairs of a step; lanes that end up with the same one
    constexpr int GPW = 32 / LPK;                          // lane groups per warp
    constexpr int NG = (kDecodeThreads / 32) * GPW;        // lane groups per block
    static_assert(V <= LPK && (V & (V - 1)) == 0, "a lane for every pair");
    extern __shared__ __align__(16) float smem[];          // the ring; the merge's records afterwards

    const int b = blockIdx.z;
    const int group = p.n_heads / p.n_kv_heads;
    const int g = blockIdx.y / p.n_sub, sub = blockIdx.y - g * p.n_sub;
    const int h0 = g * group + sub * GP;
    const int nh = (group - sub * GP) < GP ? (group - sub * GP) : GP;
    pdl_wait();
    pdl_launch();
    const bool counts = CLUSTER && blockIdx.x == 0 && blockIdx.y == 0 && b == 0;  // (last of all: off every row's path)
    const int nk = p.n_keys ? p.n_keys[b] : p.n_keys_all;
    if (nk < 1 || nk > p.n_ctx) {
        // decode.attnStep refuses an empty prefix (src/decode.zig:350); on the device the refusal is a NaN row plus
        // a count the host can read.  (Two launches: the combine kernel writes the rows.)
        if (CLUSTER && blockIdx.x == 0) {
            for (int i = threadIdx.x; i < nh * p.dim; i += kDecodeThreads) p.out[((long long)b * p.n_heads + h0) * p.dim + i] = __int_as_float(0x7fc00000);
            if (p.lse && threadIdx.x < nh) p.lse[(long long)b * p.n_heads + h0 + threadIdx.x] = __int_as_float(0x7fc00000);
        }
        if (counts) count_bad_sequences(p);
        return;  // (the whole cluster)
    }
    const int chunk = CLUSTER ? (nk + p.cluster - 1) / p.cluster : p.chunk;
    const int c0 = blockIdx.x * chunk;
    if (!CLUSTER && c0 >= nk) return;
    const int c1 = (c0 + chunk < nk) ? c0 + chunk : nk;  // (a cluster's last blocks may have no key: c0 >= c1)

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int li = lane % LPK;
    const int gi = warp * GPW + lane / LPK;
    const int dim = p.dim, n_chunks4 = dim >> 2;
    const long long kvw = (long long)p.n_kv_heads * dim;
    const long long first = b * p.cache_batch_stride + (long long)(c0 + gi) * kvw + (long long)g * dim + li * 4;
    const float *kb = p.k_cache + first, *vb = p.v_cache + first;
    const int n_mine = c1 - c0 - gi;  // this lane group's keys are the i < n_mine with i a multiple of NG
    const int n_steps = c1 > c0 ? (c1 - c0 + NG * U - 1) / (NG * U) : 0;
    const float4 *ring = reinterpret_cast<const float4 *>(smem) + threadIdx.x;  // [S][U][NCH][2][threads]
    const uint32_t ring_u32 = (uint32_t)__cvta_generic_to_shared(ring);
    const auto fetch = [&](int step) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = (step * U + u) * NG;
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const bool in = i < n_mine && li + LPK * c < n_chunks4;
                const long long off = (long long)i * kvw + LPK * c * 4;
                const uint32_t dst = ring_u32 + (uint32_t)((((step % S) * U + u) * NCH + c) * 2 * kDecodeThreads * 16);
                copy16_async(dst, in ? kb + off : p.k_cache, in);
                copy16_async(dst + kDecodeThreads * 16, in ? vb + off : p.v_cache, in);
            }
        }
    };
#pragma unroll
    for (int i = 0; i < S - 1; ++i) {
        if (i < n_steps) fetch(i);
        copy_async_commit();
    }

    // This lane's slices of the group's query rows, pre-multiplied by log2(e)/sqrt(dim).
    float4 qr[GP][NCH];
#pragma unroll
    for (int hh = 0; hh < GP; ++hh)
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const int ch = li + LPK * c;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (hh < nh && ch < n_chunks4) {
                x = *reinterpret_cast<const float4 *>(p.q + ((long long)b * p.n_heads + h0 + hh) * dim +
                                                      ch * 4);
                x.x *= p.scale_log2, x.y *= p.scale_log2, x.z *= p.scale_log2, x.w *= p.scale_log2;
            }
            qr[hh][c] = x;
        }

    // of the pair this lane ends up with, key `own / GP` of a step and head `own % GP`:
    const int own_key = (li / SP) / GP * NG;
    float m_own = kNoKey, l_own = 0.f;
    float4 acc[GP][NCH];
#pragma unroll
    for (int hh = 0; hh < GP; ++hh)
#pragma unroll
        for (int c = 0; c < NCH; ++c) acc[hh][c] = make_float4(0.f, 0.f, 0.f, 0.f);

    // The trip count is the same for every lane of the block (the shuffles below name the
    // whole warp); a lane group whose keys run out early carries -inf scores instead.
    for (int step = 0; step < n_steps; ++step) {
        copy_async_wait<S - 2>();
        if (step + S - 1 < n_steps) fetch(step + S - 1);  // into the slot that step - 1 has used up
        copy_async_commit();
        const float4 *slot = ring + (step % S) * (U * NCH * 2 * kDecodeThreads);
        float d[V];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int hh = 0; hh < GP; ++hh) d[u * GP + hh] = 0.f;
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const float4 kf = slot[(u * NCH + c) * 2 * kDecodeThreads];
#pragma unroll
                for (int hh = 0; hh < GP; ++hh) {
                    float &x = d[u * GP + hh];
                    x = fmaf(kf.x, qr[hh][c].x, x), x = fmaf(kf.y, qr[hh][c].y, x);
                    x = fmaf(kf.z, qr[hh][c].z, x), x = fmaf(kf.w, qr[hh][c].w, x);
                }
            }
        }
#pragma unroll
        for (int n = V / 2, off = LPK / 2; off > 0; n >>= 1, off >>= 1) {
            if (n > 0) {
                const bool up = (lane & off) != 0;
#pragma unroll
                for (int i = 0; i < n; ++i) {
                    const float send = up ? d[i] : d[i + n], keep = up ? d[i + n] : d[i];
                    d[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            } else {
                d[0] += __shfl_xor_sync(0xffffffffu, d[0], off);
            }
        }
        const float sc = (step * U * NG + own_key < n_mine) ? d[0] : -INFINITY;
        if (__any_sync(0xffffffffu, sc > m_own + kDecodeLazy)) {
            float mx = fmaxf(m_own, sc);
#pragma unroll
            for (int off = SP * GP; off < LPK; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            const float f = ex2(m_own - mx);
            l_own *= f, m_own = mx;
#pragma unroll
            for (int hh = 0; hh < GP; ++hh) {
                const float fh = __shfl_sync(0xffffffffu, f, hh * SP, LPK);
#pragma unroll
                for (int c = 0; c < NCH; ++c) acc[hh][c].x *= fh, acc[hh][c].y *= fh, acc[hh][c].z *= fh, acc[hh][c].w *= fh;
            }
        }
        const float p_own = ex2(sc - m_own);  // exp2(-inf) = 0 for absent keys
        l_own += p_own;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float pe[GP];
#pragma unroll
            for (int hh = 0; hh < GP; ++hh) pe[hh] = __shfl_sync(0xffffffffu, p_own, (u * GP + hh) * SP, LPK);
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const float4 vf = slot[((u * NCH + c) * 2 + 1) * kDecodeThreads];
#pragma unroll
                for (int hh = 0; hh < GP; ++hh) {
                    acc[hh][c].x = fmaf(pe[hh], vf.x, acc[hh][c].x), acc[hh][c].y = fmaf(pe[hh], vf.y, acc[hh][c].y);
                    acc[hh][c].z = fmaf(pe[hh], vf.z, acc[hh][c].z), acc[hh][c].w = fmaf(pe[hh], vf.w, acc[hh][c].w);
                }
            }
        }
    }
    copy_async_wait<0>();
    // every lane of the group learns every head's maximum and denominator
#pragma unroll
    for (int off = SP * GP; off < LPK; off <<= 1) l_own += __shfl_xor_sync(0xffffffffu, l_own, off);
    float m[GP], l[GP];
#pragma unroll
    for (int hh = 0; hh < GP; ++hh) {
        const float mo = __shfl_sync(0xffffffffu, m_own, hh * SP, LPK);
        m[hh] = mo == kNoKey ? -INFINITY : mo;
        l[hh] = __shfl_sync(0xffffffffu, l_own, hh * SP, LPK);
    }
    __syncthreads();  // the ring's slots are the merge's records from here on

    // Merge the lane groups of a warp.  A group that saw no key has m = -inf, l = 0.
#pragma unroll
    for (int off = LPK; off < 32; off <<= 1) {
#pragma unroll
        for (int hh = 0; hh < GP; ++hh) {
            const float mo = __shfl_xor_sync(0xffffffffu, m[hh], off);
            const float lo = __shfl_xor_sync(0xffffffffu, l[hh], off);
            const float mx = fmaxf(m[hh], mo);
            const float cs = (m[hh] == -INFINITY) ? 0.f : ex2(m[hh] - mx);
            const float co = (mo == -INFINITY) ? 0.f : ex2(mo - mx);
            l[hh] = l[hh] * cs + lo * co;
            m[hh] = mx;
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                float4 o;
                o.x = __shfl_xor_sync(0xffffffffu, acc[hh][c].x, off);
                o.y = __shfl_xor_sync(0xffffffffu, acc[hh][c].y, off);
                o.z = __shfl_xor_sync(0xffffffffu, acc[hh][c].z, off);
                o.w = __shfl_xor_sync(0xffffffffu, acc[hh][c].w, off);
                acc[hh][c].x = acc[hh][c].x * cs + o.x * co;
                acc[hh][c].y = acc[hh][c].y * cs + o.y * co;
                acc[hh][c].z = acc[hh][c].z * cs + o.z * co;
                acc[hh][c].w = acc[hh][c].w * cs + o.w * co;
            }
        }
    }

    // Merge the warps through shared memory: [warp][head][dim + 4].
    constexpr int NW = kDecodeThreads / 32;
    const int rec = dim + 4;  // [0] max, [1] denominator, [4 ..] accumulators (16-byte aligned)
    if (lane < LPK) {
#pragma unroll
        for (int hh = 0; hh < GP; ++hh) {
            float *dst = smem + (warp * GP + hh) * rec;
#pragma unroll
            for (int c = 0; c < NCH; ++c) {
                const int ch = li + LPK * c;
                if (ch < n_chunks4) *reinterpret_cast<float4 *>(dst + 4 + ch * 4) = acc[hh][c];
            }
            if (lane == 0) dst[0] = m[hh], dst[1] = l[hh];
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < nh * dim; idx += kDecodeThreads) {
        const int hh = idx / dim, j = idx - hh * dim;
        float mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < NW; ++w) mx = fmaxf(mx, smem[(w * GP + hh) * rec]);
        float lsum = 0.f, a = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const float *src = smem + (w * GP + hh) * rec;
            const float cw = (src[0] == -INFINITY) ? 0.f : ex2(src[0] - mx);
            lsum = fmaf(src[1], cw, lsum);
            a = fmaf(src[4 + j], cw, a);
        }
        if (CLUSTER) {
            float *blk = smem + NW * GP * rec + hh * rec;  // the block's own sums, for its cluster to read
            blk[4 + j] = a;
            if (j == 0) blk[0] = mx, blk[1] = lsum;
        } else {
            const long long slot = ((long long)b * p.n_heads + h0 + hh) * p.max_chunks + blockIdx.x;
            p.part_acc[slot * dim + j] = a;
            if (j == 0) p.part_ml[slot] = make_float2(mx, lsum);
        }
    }
    if (!CLUSTER) return;
    cluster_arrive();
    cluster_wait();
    const int cs = p.cluster;
    const uint32_t blk0 = (uint32_t)__cvta_generic_to_shared(smem + NW * GP * rec);
    for (int idx = blockIdx.x * kDecodeThreads + threadIdx.x; idx < nh * dim; idx += cs * kDecodeThreads) {
        const int hh = idx / dim, j = idx - hh * dim;
        const uint32_t at = blk0 + (uint32_t)(hh * rec) * 4u;
        float mr[kMaxCluster], lr[kMaxCluster], ar[kMaxCluster], mx = -INFINITY;  // (block 0 has keys: the maximum is finite)
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) {  // all of them on their way at once
            mr[r] = r < cs ? ld_cluster(at, r) : -INFINITY;
            lr[r] = r < cs ? ld_cluster(at + 4u, r) : 0.f;
            ar[r] = r < cs ? ld_cluster(at + 4u * (4 + j), r) : 0.f;
        }
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) mx = fmaxf(mx, mr[r]);
        float lsum = 0.f, acc_j = 0.f;
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) {
            const float w = (mr[r] == -INFINITY) ? 0.f : ex2(mr[r] - mx);
            lsum = fmaf(lr[r], w, lsum);
            acc_j = fmaf(ar[r], w, acc_j);
        }
        const long long row = (long long)b * p.n_heads + h0 + hh;
        p.out[row * dim + j] = acc_j / lsum;
        if (p.lse && j == 0) p.lse[row] = (mx + log2f(lsum)) * kLn2;
    }
    cluster_arrive();  // nobody's shared memory goes away while others read it
    if (counts) count_bad_sequences(p);
    cluster_wait();
}

// Log-sum-exp combine of a sequence's chunks.  grid (n_heads, batch), block 128.
__global__ void __launch_bounds__(128) decode_combine_kernel(const DecodeParams p) {
    const int h = blockIdx.x, b = blockIdx.y;
    pdl_wait();
    pdl_launch();
    const bool counts = h == 0 && b == 0;
    const int nk = p.n_keys ? p.n_keys[b] : p.n_keys_all;
    float *orow = p.out + ((long long)b * p.n_heads + h) * p.dim;
    if (nk < 1 || nk > p.n_ctx) {
        for (int j = threadIdx.x; j < p.dim; j += blockDim.x) orow[j] = __int_as_float(0x7fc00000);
        if (threadIdx.x == 0 && p.lse) p.lse[(long long)b * p.n_heads + h] = __int_as_float(0x7fc00000);
        if (counts) count_bad_sequences(p);
        return;
    }
    const int nchunks = (nk + p.chunk - 1) / p.chunk;
    const long long slot0 = ((long long)b * p.n_heads + h) * p.max_chunks;
    float mx = -INFINITY;
    for (int c = threadIdx.x & 31; c < nchunks; c += 32) mx = fmaxf(mx, p.part_ml[slot0 + c].x);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    float lsum = 0.f;
    for (int c = threadIdx.x & 31; c < nchunks; c += 32) {
        const float2 ml = p.part_ml[slot0 + c];
        lsum = fmaf(ml.y, ex2(ml.x - mx), lsum);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
    const float inv = 1.f / lsum;
    for (int j = threadIdx.x; j < p.dim; j += blockDim.x) {
        float a = 0.f;
#pragma unroll 8
        for (int c = 0; c < nchunks; ++c)
            a = fmaf(p.part_acc[(slot0 + c) * p.dim + j], ex2(p.part_ml[slot0 + c].x - mx), a);
        orow[j] = a * inv;
    }
    if (p.lse && threadIdx.x == 0)
        p.lse[(long long)b * p.n_heads + h] = (mx + log2f(lsum)) * kLn2;
    if (counts) count_bad_sequences(p);
}

// kv_cache.Layer.append for a batch (src/kv_cache.zig:88-95).  grid (batch), block 256.  VEC: four floats at a time (the
// rows of both caches and of the new rows start on 16-byte boundaries).
template <bool VEC>
__global__ void __launch_bounds__(256) kv_append_kernel(float *k_cache, float *v_cache, int *n_keys, const float *k_new,
                                                        const float *v_new, int *full_count, int n_ctx, int width) {
    const int b = blockIdx.x;
    pdl_wait();
    pdl_launch();
    const int len = n_keys[b];
    if (len < 0 || len >= n_ctx) {  // Error.Full: nothing is written, nothing advances
        if (threadIdx.x == 0 && full_count) atomicAdd(full_count, 1);
        return;
    }
    float *kd = k_cache + ((long long)b * n_ctx + len) * width;
    float *vd = v_cache + ((long long)b * n_ctx + len) * width;
    const float *ks = k_new + (long long)b * width, *vs = v_new + (long long)b * width;
    if (VEC) {
        for (int j = threadIdx.x * 4; j < width; j += 1024) {
            const float4 kx = *reinterpret_cast<const float4 *>(ks + j), vx = *reinterpret_cast<const float4 *>(vs + j);
            *reinterpret_cast<float4 *>(kd + j) = kx, *reinterpret_cast<float4 *>(vd + j) = vx;
        }
    } else {
        for (int j = threadIdx.x; j < width; j += 256) kd[j] = ks[j], vd[j] = vs[j];
    }
    __syncthreads();
    if (threadIdx.x == 0) n_keys[b] = len + 1;
}

// ---- host side ---------------------------------------------------------------

struct DecodePlan {
    int lpk, nch, gp, n_sub, chunk, max_chunks;
    int cluster;  // blocks per (sequence, KV head, pass) in the one-launch form; 0: two launches
    size_t ml_bytes, acc_bytes, total_bytes;
};

// The split is a pure function of the shape and of the current device's SM count, so the
// workspace-size query and the launch agree (both made with the same device current).  The
// chunk is as large as keeps roughly eight blocks an SM in the launch, between 128 and 1024
// keys.  Without a device (a size query on a machine with none) the
// count of a B200, 148, stands in.
inline DecodePlan decode_plan(int batch, int n_ctx, int n_heads, int n_kv_heads, int dim) {
    DecodePlan pl{};
    const int group = n_heads / n_kv_heads;
    pl.gp = group >= 3 ? 4 : group;
    pl.n_sub = (group + pl.gp - 1) / pl.gp;
    const int chunks4 = dim / 4;
    pl.lpk = chunks4 <= 8 ? 8 : 16;
    pl.nch = (chunks4 + pl.lpk - 1) / pl.lpk;
    const long long units = (long long)batch * n_kv_heads * pl.n_sub;
    const DeviceInfo *di = device_info();
    const int sms = di && di->sm_count > 0 ? di->sm_count : 148;
    const long long target_blocks = 8LL * sms;
    long long want = (target_blocks + units - 1) / units;
    if (want < 1) want = 1;
    long long chunk = (n_ctx + want - 1) / want;
    chunk = (chunk + 63) / 64 * 64;
    if (chunk < 128) chunk = 128;
    if (chunk > 1024) chunk = 1024;
    pl.chunk = (int)chunk;
    pl.max_chunks = (n_ctx + pl.chunk - 1) / pl.chunk;
    // One launch where clusters of at most eight blocks find an SM slot each at once and a block's share stays below 768
    // keys; 32/8 heads of 128, us a call: one sequence, 512 keys 6.9 against 12.9, 2048 keys 11.1
    // against 18.4, 8192 keys 39.4 against 35.6; four sequences, 2048 keys 19.4 against 30.7; sixteen (a second wave of
    // clusters), 512 keys 34.0 against 27.5.  (Clusters of sixteen start late: 36.7 where eight take 19.4.)
    // Where an SM holds one block only, clusters of up to two waves serve what one wave's share is too long for: 32/8 heads
    // of 256, four sequences of 4096 keys 75 against 93, sixteen of 1024 keys 56 against 75.  What fits one wave is better
    // off with it: four of 1024 keys 16.8 in one wave, 33.2 in two; eight of 256 keys 12.4 and 17.3.
    const int per_sm = decode_blocks_per_sm(pl.nch, pl.gp);
    const auto clusters_in = [&](long long slots) -> int {
        long long cs = 1;
        while (cs < kMaxCluster && 2 * cs * units <= slots && n_ctx > 64 * cs) cs *= 2;
        return cs * units <= slots && n_ctx <= 768 * cs ? (int)cs : 0;
    };
    pl.cluster = clusters_in((long long)per_sm * sms);
    if (pl.cluster == 0 && per_sm == 1) pl.cluster = clusters_in(2LL * sms);
    pl.ml_bytes = (size_t)batch * n_heads * pl.max_chunks * sizeof(float2);
    pl.ml_bytes = (pl.ml_bytes + 255) / 256 * 256;
    pl.acc_bytes = (size_t)batch * n_heads * pl.max_chunks * dim * sizeof(float);
    pl.total_bytes = kDecodeHeaderBytes + pl.ml_bytes + pl.acc_bytes;
    return pl;
}

template <int LPK, int NCH, int GP>
inline int launch_decode_inst(const DecodeParams &p, cudaStream_t stream) {
    using Cfg = DecodeCfg<LPK, NCH, GP>;
    size_t smem = (size_t)Cfg::kStages * Cfg::kStageBytes;
    const size_t merge = (size_t)(kDecodeThreads / 32 + 1) * GP * (p.dim + 4) * sizeof(float);
    if (smem < merge) smem = merge;
    const auto kernel = p.cluster ? decode_splitk_kernel<LPK, NCH, GP, true> : decode_splitk_kernel<LPK, NCH, GP, false>;
    if (optin_smem((const void *)kernel, smem)) return 1;
    const dim3 grid((unsigned)(p.cluster ? p.cluster : p.max_chunks), (unsigned)(p.n_kv_heads * p.n_sub), (unsigned)p.batch);
    if (p.cluster) return launch_pdl_cluster("decode_splitk_kernel", kernel, grid, dim3(kDecodeThreads), smem, stream, p.cluster, p);
    return launch_pdl("decode_splitk_kernel", kernel, grid, dim3(kDecodeThreads), smem, stream, p);
}

template <int LPK, int NCH>
inline int launch_decode_gp(const DecodeParams &p, int gp, cudaStream_t stream) {
    switch (gp) {
        case 1: return launch_decode_inst<LPK, NCH, 1>(p, stream);
        case 2: return launch_decode_inst<LPK, NCH, 2>(p, stream);
        default: return launch_decode_inst<LPK, NCH, 4>(p, stream);
    }
}

// One launch, or the split-K pass followed by the combine, on `stream`.
inline int launch_decode(DecodeParams p, const DecodePlan &pl, void *workspace, cudaStream_t stream) {
    char *ws = static_cast<char *>(workspace);
    p.bad_count = reinterpret_cast<int *>(ws);
    p.part_ml = reinterpret_cast<float2 *>(ws + kDecodeHeaderBytes);
    p.part_acc = reinterpret_cast<float *>(ws + kDecodeHeaderBytes + pl.ml_bytes);
    p.chunk = pl.chunk, p.max_chunks = pl.max_chunks, p.n_sub = pl.n_sub, p.cluster = pl.cluster;
    int rc;
    if (pl.lpk == 8) rc = launch_decode_gp<8, 1>(p, pl.gp, stream);
    else if (pl.nch == 1) rc = launch_decode_gp<16, 1>(p, pl.gp, stream);
    else if (pl.nch == 2) rc = launch_decode_gp<16, 2>(p, pl.gp, stream);
    else if (pl.nch == 3) rc = launch_decode_gp<16, 3>(p, pl.gp, stream);
    else rc = launch_decode_gp<16, 4>(p, pl.gp, stream);
    if (rc) return rc;
    g_last_path = "decode-splitk";
    if (pl.cluster) return 0;
    const dim3 cgrid((unsigned)p.n_heads, (unsigned)p.batch);
    return launch_pdl("decode_combine_kernel", decode_combine_kernel, cgrid, dim3(128), 0, stream, p);
}

}  // namespace zt
