// The pre-pass of the tensor-core kernels: f32 tensors -> f16 hi/lo operand planes with a power-of-two scale per
// (sequence, group of heads), and beside them what the backward wants to know about the rows of dout.
//
// A forward's are k and v (its kernels split the query rows themselves); a backward's dout and q, and k and v where the forward has not kept
// them.  One launch where a block or a cluster holds a (sequence, group)'s rows (pass_one_kernel, the forms of pass_planes_kernel that
// hold them, pass_backward_kernel), else two for all tensors of a call, bound by HBM (or, for small calls, by launch latency):
//   pass_stats_kernel    reads every tensor once.  Per block: max |x| and, where asked, the largest row norm; per row of
//                        dout its norm and delta = sum_j dout out.  A block leaves its two maxima in a slot of its own
//                        (no atomics and nothing to clear beforehand).
//   pass_planes_kernel   reads the slots of its (sequence, group) -- at most 1024 of them --, publishes the maxima for
//                        the attention kernels, and writes the planes (rotating q and k on the way where rope is asked
//                        for), the row-scaled copy of q's planes for dK, and the zeros of outputs that are summed in memory.
// Both work on units, one head of one row, held by 8, 16 or 32 lanes.  A lane of the first launch has three units under way, of
// the second four (two where it holds two or three chunks of one).  A block's units belong to one (sequence, group), of which its
// blocks take turns: blocks that run together read and write one stretch of memory, not a stretch each (the first launch of a step at
// T 4096, heads of 128, when it read q too: 460 us, with the turns 417).  The split into blocks is in pass_add.
// Us of a step's pre-passes, forward and backward with k and v kept: batch 8, T 512, 32/8 heads of 64 66; T 1024, heads of 256,
// 410 (its q goes into two pairs of planes); T 4096, heads of 128, 830 for 4.6 GB read and written, 700 at the copy rate.
#pragma once

#include <cuda_fp16.h>

#include "rope_kernels.cuh"
#include "zt_common.cuh"

namespace zt {
namespace tcb {

// ---- scaling --------------------------------------------------------------------------------------
// The power of two that moves a block's largest magnitude into [2^14, 2^15).  `bits` is the f32
// bit pattern of max |x| (non-negative, so it orders like an integer).
__host__ __device__ inline float block_mult(uint32_t bits) {
    const int ex = (int)((bits >> 23) & 0xff);  // biased exponent: |x| in [2^(ex-127), 2^(ex-126))
    if (ex == 0 || ex == 0xff) return 1.0f;      // zero/subnormal block, or inf/nan: leave alone
    int e = 14 - (ex - 127);                     // |x| * 2^e in [2^14, 2^15)
    if (e > 126) e = 126;
    if (e < -126) e = -126;
    uint32_t out = (uint32_t)(e + 127) << 23;
#if defined(__CUDA_ARCH__)
    return __uint_as_float(out);
#else
    float f;
    memcpy(&f, &out, 4);
    return f;
#endif
}
// pow2_for(x, top): the power of two c with x c in [2^(top-1), 2^top); 1 when x is zero or not finite.
__device__ __forceinline__ float pow2_for(float x, int top) {
    if (!(x > 0.f) || !(x < 3.0e38f)) return 1.0f;
    int e;
    frexpf(x, &e);  // x = m 2^e, m in [0.5, 1)
    int k = top - e;
    k = k > 120 ? 120 : (k < -120 ? -120 : k);
    return __uint_as_float((uint32_t)(k + 127) << 23);
}
// Row t's scale of dS (cq) and what divides row t of the second copy of Q (1 / rel): both powers of two.
constexpr float kRowBoostMax = 4096.f;  // a row's scale is at most this many times the group's smallest
__device__ __forceinline__ float ds_group_scale(uint32_t rnmax_bits, uint32_t vnmax_bits) {
    return pow2_for(2.02f * __uint_as_float(rnmax_bits) * __uint_as_float(vnmax_bits), 14);
}
__device__ __forceinline__ void ds_row_scale(float rnorm_t, uint32_t rnmax_bits, uint32_t vnmax_bits, float &cq, float &rel) {
    const float cmin = ds_group_scale(rnmax_bits, vnmax_bits);
    const float x = 2.02f * rnorm_t * __uint_as_float(vnmax_bits);
    float c = (x > 0.f && x < 3.0e38f) ? pow2_for(x, 14) : cmin;
    c = fminf(fmaxf(c, cmin), cmin * kRowBoostMax);
    if (!(c < 3.0e38f)) c = cmin;
    cq = c;
    rel = cmin / c;
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// Two f32 operations an instruction, each rounded as the single one is.
__device__ __forceinline__ uint64_t pair2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpair2(uint64_t r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pair2(a.x, a.y)), "l"(pair2(b.x, b.y)), "l"(pair2(c.x, c.y)));
    return unpair2(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pair2(a.x, a.y)), "l"(pair2(b.x, b.y)));
    return unpair2(r);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pair2(a.x, a.y)), "l"(pair2(b.x, b.y)));
    return unpair2(r);
}
__device__ __forceinline__ float2 floats2(uint32_t a, uint32_t b) { return make_float2(__uint_as_float(a), __uint_as_float(b)); }
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// x with its magnitude cut to `bound` (> 0); the bound itself for a NaN
__device__ __forceinline__ float clamp_abs(float x, float bound) {
    float r;
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(bound));
    return r;
}
// v -> packed h pair and packed l pair, two values an instruction but for the way back
__device__ __forceinline__ void split_pack(float2 v, uint32_t &hw, uint32_t &lw) {
    const __half2 hh = __floats2half2_rn(v.x, v.y);
    const float2 lo = fma2(__half22float2(hh), make_float2(-1.f, -1.f), v);
    hw = *reinterpret_cast<const uint32_t *>(&hh);
    lw = pack_half2(lo.x, lo.y);
}
__device__ __forceinline__ void split_pack(float a, float b, uint32_t &hw, uint32_t &lw) { split_pack(make_float2(a, b), hw, lw); }

// ---- the two launches -------------------------------------------------------------------------------
constexpr int kPrepassMaxGroups = 256;
constexpr int kPassThreads = 256, kStatsStages = 4, kPassUnroll = 4;
constexpr int kPassTargetBlocks = 2048, kPassMaxSlots = 1024, kPassMaxTensors = 5;
constexpr int kFillPerBlock = 4096;  // float4

struct PassTensor {
    const float *x;          // [batch][rows][heads * dim]
    const float *o;          // with delta: the tensor it is formed with
    float *delta, *rnorm;    // [batch][rows][heads], or null
    __half *planes;          // [2][batch][rows][heads * pd], or null
    uint2 *part;             // [batch * groups][slots] (max |x|, largest row norm) as f32 bit patterns; null: amax is known already
    uint32_t *amax, *nmax;   // [batch * groups]: where the maxima are published; nmax null: not wanted
    uint32_t *clear;         // [batch * groups] words set to zero, or null
    const float2 *rope;      // null, or the (cos, sin) table [rows][dim / 2]: x is rotated on its way into the planes
    // the planes with row t times rel(t) (ds_row_scale, from rnorm and the largest row norms of dout and v), or null; together with `planes`
    // above 128 columns only
    __half *qs;
    const uint2 *dn_part, *vn_part;  // dout's slots; v's, or null: v's norms are published already
    const uint32_t *vn_final;
    int dn_slots, vn_slots;
    int batch, rows, heads, group;  // heads per row, heads per group
    uint32_t per_head;              // what a unit's index is divided by `group` with (pass_row)
    int slots;                      // blocks per (sequence, group)
    int first;                      // first block of this tensor
};
struct PassArgs {
    PassTensor t[kPassMaxTensors];
    float4 *fill[3];
    long long fill_n4[3];
    int fill_first[4];  // first block of each region; [n_fill]: one past the last
    int n, n_stats, n_fill, dim, pd;  // dim: columns of a head in the tensors; pd: in the planes (plane_dim)
    int cluster, per;                 // of the one-launch forms: blocks per (sequence, group); units that a lane group of a backward's takes
    int q_units;  // of a forward: rows times heads of a (sequence, group)'s queries, which no launch here reads (see pass_takes_one)
};

// The row of a (sequence, group)'s unit u.  (A product with 2^32 / group rounded up, which is exact where pass_add has found it so: two divisions a
// step were a fifth of the first launch's time: us, batch 8, T 4096, 32/8 heads of 128, 345 -> 279, the second launch 611 -> 556.)
__host__ __device__ __forceinline__ int pass_row(const PassTensor &t, int u) {
    return t.per_head ? (int)(((unsigned long long)(uint32_t)u * t.per_head) >> 32) : t.group == 1 ? u : u / t.group;
}
struct PassUnit {  // where a block stands
    int z, bg, slot, b, g, units;
};
__device__ __forceinline__ PassUnit pass_locate(const PassArgs &a, int n, int blk) {
    PassUnit w;
    w.z = 0;
    while (w.z + 1 < n && blk >= a.t[w.z + 1].first) ++w.z;
    const PassTensor &t = a.t[w.z];
    const int groups = t.heads / t.group, i = blk - t.first;
    // (the groups of the same rows are neighbours: blocks that run together cover whole rows)
    const int rest = i / groups;
    w.g = i - rest * groups, w.b = rest / t.slots, w.slot = rest - w.b * t.slots;
    w.bg = w.b * groups + w.g;
    w.units = t.rows * t.group;
    return w;
}

// LP lanes hold a unit, NC float4 each.  The loads run kStatsStages - 1 units ahead through slots of shared memory
// that belong to one thread each (so nothing but the thread's own copies is waited for): held in registers instead,
// the loads of a step would stall on the arithmetic of the step before (heads of 256, batch 8, T 1024: 4.1 TB/s against 5.4).
// O4: the tensor that dout is multiplied with starts on a 4-byte boundary only (of a call's tensors it alone may, because
// nothing but its row sums is wanted).  A variant of its own: asked per copy it cost every backward 0.4 us.
template <int LP, int NC, bool O4>
__global__ void __launch_bounds__(kPassThreads) pass_stats_kernel(const __grid_constant__ PassArgs a) {
    constexpr int NG = kPassThreads / LP, S = kStatsStages;
    extern __shared__ __align__(16) float4 ring[];  // [S][NC][2][kPassThreads]
    __shared__ float red[2][kPassThreads / 32];
    const PassUnit w = pass_locate(a, a.n_stats, (int)blockIdx.x);
    const PassTensor &t = a.t[w.z];
    const int gi = threadIdx.x / LP, li = threadIdx.x % LP, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool rows_out = t.delta != nullptr, norms = rows_out || t.nmax != nullptr;
    const int n4 = a.dim >> 2, group = t.group, heads = t.heads;
    const long long first = (long long)w.b * t.rows * heads + w.g * group;  // the (sequence, group)'s first unit
    const float4 *xb = reinterpret_cast<const float4 *>(t.x) + first * n4 + li;
    const float4 *ob = reinterpret_cast<const float4 *>(rows_out ? t.o : t.x) + first * n4 + li;
    const uint32_t slot0 = (uint32_t)__cvta_generic_to_shared(ring + threadIdx.x);
    const int stride = t.slots * NG, n_steps = (w.units - w.slot * NG + stride - 1) / stride;
    const auto place = [&](int step) -> int {  // the unit's index within the (sequence, group), or -1
        const int u = step * stride + w.slot * NG + gi;
        return u < w.units ? pass_row(t, u) * (heads - group) + u : -1;  // r heads + (u - r group)
    };
    const auto fetch = [&](int step) {
        const int at = place(step);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const bool in = step < n_steps && at >= 0 && li + LP * c < n4;
            const long long off = in ? (long long)at * n4 + LP * c : 0;
            const uint32_t dst = slot0 + (uint32_t)(((step % S) * NC + c) * 2 * kPassThreads * 16);
            copy16_async(dst, xb + off, in);
            if (rows_out && O4) copy16_async_by4(dst + kPassThreads * 16, ob + off, in);
            else if (rows_out) copy16_async(dst + kPassThreads * 16, ob + off, in);
        }
        copy_async_commit();
    };
    pdl_wait();
    pdl_launch();
#pragma unroll
    for (int i = 0; i < S - 1; ++i) fetch(i);
    float amax = 0.f, nmax = 0.f;
    for (int step = 0; step < n_steps; ++step) {
        copy_async_wait<S - 2>();
        float sq = 0.f, de = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const float4 *at = ring + ((step % S) * NC + c) * 2 * kPassThreads + threadIdx.x;
            const float4 x = at[0];
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));
            sq = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, sq))));
            if (rows_out) {
                const float4 o = at[kPassThreads];
                de = fmaf(x.x, o.x, fmaf(x.y, o.y, fmaf(x.z, o.z, fmaf(x.w, o.w, de))));
            }
        }
        fetch(step + S - 1);
        if (!norms) continue;
#pragma unroll
        for (int off = LP / 2; off > 0; off >>= 1) {
            sq += __shfl_xor_sync(0xffffffffu, sq, off);
            if (rows_out) de += __shfl_xor_sync(0xffffffffu, de, off);
        }
        const float norm = sqrtf(sq);
        nmax = fmaxf(nmax, norm);
        const int at = place(step);
        if (rows_out && li == 0 && at >= 0) t.delta[first + at] = de, t.rnorm[first + at] = norm;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        nmax = fmaxf(nmax, __shfl_xor_sync(0xffffffffu, nmax, off));
    }
    if (lane == 0) red[0][warp] = amax, red[1][warp] = nmax;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 1; i < kPassThreads / 32; ++i) amax = fmaxf(amax, red[0][i]), nmax = fmaxf(nmax, red[1][i]);
        t.part[(long long)w.bg * t.slots + w.slot] = make_uint2(__float_as_uint(amax), __float_as_uint(nmax));
    }
}

// The maxima a block of the second launch needs, from the slots the first one left: its own tensor's and, for the row-scaled
// copy, the largest row norms of dout and v.  (f32 bit patterns of non-negative numbers order like integers.)
struct PassTops {
    uint32_t amax, nmax, dn, vn;
};
__device__ __forceinline__ PassTops pass_tops(const PassTensor &t, int bg, uint4 *red) {
    uint4 m = make_uint4(0u, 0u, 0u, 0u);
    if (t.part == nullptr) {
        m.x = t.amax[bg];
    } else {
        const uint2 *part = t.part + (long long)bg * t.slots;
        for (int i = threadIdx.x; i < t.slots; i += kPassThreads) {
            const uint2 v = part[i];
            m.x = max(m.x, v.x), m.y = max(m.y, v.y);
        }
    }
    if (t.qs) {
        const uint2 *part = t.dn_part + (long long)bg * t.dn_slots;
        for (int i = threadIdx.x; i < t.dn_slots; i += kPassThreads) m.z = max(m.z, part[i].y);
        if (t.vn_part) {
            const uint2 *vp = t.vn_part + (long long)bg * t.vn_slots;
            for (int i = threadIdx.x; i < t.vn_slots; i += kPassThreads) m.w = max(m.w, vp[i].y);
        } else {
            m.w = t.vn_final[bg];
        }
    }
    m.x = __reduce_max_sync(0xffffffffu, m.x), m.y = __reduce_max_sync(0xffffffffu, m.y);
    m.z = __reduce_max_sync(0xffffffffu, m.z), m.w = __reduce_max_sync(0xffffffffu, m.w);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPassThreads / 32; ++i) {
        const uint4 v = red[i];
        m.x = max(m.x, v.x), m.y = max(m.y, v.y), m.z = max(m.z, v.z), m.w = max(m.w, v.w);
    }
    return PassTops{m.x, m.y, m.z, m.w};
}

// Four elements times m into the planes at `hi`.
__device__ __forceinline__ void store_split4(__half *hi, long long plane, float4 v, float m) {
    uint2 hw, lw;
    split_pack(v.x * m, v.y * m, hw.x, lw.x);
    split_pack(v.z * m, v.w * m, hw.y, lw.y);
    *reinterpret_cast<uint2 *>(hi) = hw, *reinterpret_cast<uint2 *>(hi + plane) = lw;
}

// Block blk's part of the zeros of outputs that are summed in memory.
template <int THREADS>
__device__ __forceinline__ void pass_fill_block(const PassArgs &a, int blk) {
    int f = 0;
    while (f + 1 < a.n_fill && blk >= a.fill_first[f + 1]) ++f;
    const long long i0 = (long long)(blk - a.fill_first[f]) * kFillPerBlock;
#pragma unroll
    for (int k = 0; k < kFillPerBlock / THREADS; ++k) {
        const long long i = i0 + k * THREADS + threadIdx.x;
        if (i < a.fill_n4[f]) a.fill[f][i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// LP lanes hold a unit of the planes (pd columns), NC chunks of four columns each.
template <int LP, int NC>
__global__ void __launch_bounds__(kPassThreads, LP * NC > 32 ? 3 : 0) pass_planes_kernel(const __grid_constant__ PassArgs a) {
    constexpr int NG = kPassThreads / LP, U = (kPassUnroll + NC - 1) / NC;
    pdl_wait();
    pdl_launch();
    const int blk = (int)blockIdx.x;
    if (blk >= a.fill_first[0]) {
        pass_fill_block<kPassThreads>(a, blk);
        return;
    }
    __shared__ uint4 red[kPassThreads / 32];
    const PassUnit w = pass_locate(a, a.n, blk);
    const PassTensor &t = a.t[w.z];
    const int gi = threadIdx.x / LP, li = threadIdx.x % LP;
    const long long plane = (long long)t.batch * t.rows * t.heads * a.pd;
    const int n4 = a.dim >> 2;
    const auto locate = [&](int u, int &r) -> long long {
        r = pass_row(t, u);
        return u < w.units ? ((long long)w.b * t.rows + r) * t.heads + w.g * t.group + (u - r * t.group) : -1;
    };
    PassTops tops{};
    const auto row_rel = [&](float norm) -> float {
        float cq, rel;
        ds_row_scale(norm, tops.dn, tops.vn, cq, rel);
        return rel;
    };
    // (the first units' loads go out before the maxima are waited for: many blocks have no second units)
    const int stride = t.slots * NG * U;
    float4 x[U][NC];
    float norm[U];
    long long at[U];
    const auto load = [&](int u0) {
#pragma unroll
        for (int k = 0; k < U; ++k) {
            int r;
            at[k] = locate(u0 + k * NG + gi, r);
            norm[k] = t.qs && at[k] >= 0 ? t.rnorm[at[k]] : 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int ch = li + LP * c;
                x[k][c] = (at[k] >= 0 && ch < n4) ? __ldg(reinterpret_cast<const float4 *>(t.x + at[k] * a.dim) + ch) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    };
    int u0 = w.slot * NG * U;
    if (t.rope == nullptr) load(u0);
    tops = pass_tops(t, w.bg, red);
    if (w.slot == 0 && threadIdx.x == 0 && t.part) {
        t.amax[w.bg] = tops.amax;
        if (t.nmax) t.nmax[w.bg] = tops.nmax;
        if (t.clear) t.clear[w.bg] = 0u;
    }
    const float m = block_mult(tops.amax);
    __half *const planes = t.qs ? t.qs : t.planes;
    const bool both = LP * NC > 32 && t.qs && t.planes;  // (the wide heads' q)
    if (t.rope == nullptr) {
        for (; u0 < w.units;) {
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const float rel = t.qs ? row_rel(norm[k]) : 1.f;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const long long to = at[k] * a.pd + (li + LP * c) * 4;
                    if (at[k] < 0 || (li + LP * c) * 4 >= a.pd) continue;
                    store_split4(planes + to, plane, x[k][c], m * rel);
                    if (both) store_split4(t.planes + to, plane, x[k][c], m);
                }
            }
            u0 += stride;
            if (u0 < w.units) load(u0);
        }
        return;
    }
    // rotated: a lane of the head's lower half takes a chunk and its partner half a head on (a head's halves are
    // multiples of four wide), so that every element and every table entry is fetched once
    const int half = a.dim >> 1, h4 = half >> 2;
    for (; u0 < w.units; u0 += stride) {
#pragma unroll
        for (int k = 0; k < U; ++k) {
            int r;
            const long long at = locate(u0 + k * NG + gi, r);
            if (at < 0) break;
            const float rel = t.qs ? row_rel(t.rnorm[at]) : 1.f;
            const auto put = [&](int col, float4 v) {
                store_split4(planes + at * a.pd + col, plane, v, m * rel);
                if (both) store_split4(t.planes + at * a.pd + col, plane, v, m);
            };
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int ch = li + LP * c;
                if (ch < h4) {
                    const float4 *src = reinterpret_cast<const float4 *>(t.x + at * a.dim);
                    const float4 lo = __ldg(src + ch), hi = __ldg(src + h4 + ch);
                    const float4 *cs = reinterpret_cast<const float4 *>(t.rope + (long long)r * half) + 2 * ch;
                    float4 lr, hr;
                    rope_chunk(lo, hi, __ldg(cs), __ldg(cs + 1), lr, hr);
                    put(ch * 4, lr), put(half + ch * 4, hr);
                } else if (ch >= n4 && ch * 4 < a.pd) {
                    put(ch * 4, make_float4(0.f, 0.f, 0.f, 0.f));
                }
            }
        }
    }
}

// ---- the one launch of small forwards ---------------------------------------------------------------
// Of the one-launch forms: threads of a block, float4 that a thread of either form holds, blocks of a cluster at most.
constexpr int kOneThreads = 512, kOneMost = 16, kOneFew = 4, kOneCluster = 8;
template <int LP, int NC, int CHUNKS>
__host__ __device__ constexpr int pass_one_units() { return kOneThreads / LP * (CHUNKS / NC); }

// A block's two maxima -> its cluster's, through `slots` in global memory, one a block: behind the barrier nothing of a block is read by another, so
// that each may leave when its own work is done.
__device__ __forceinline__ void cluster_tops(uint2 *slots, int rank, int cluster, uint32_t &top, uint32_t &norm) {
    if (threadIdx.x == 0) slots[rank] = make_uint2(top, norm);
    cluster_arrive();
    cluster_wait();
    const int lane = (int)threadIdx.x & 31;
    const uint2 v = __ldcg(slots + (lane < cluster ? lane : 0));  // (from L2, where the others' words are)
    top = __reduce_max_sync(0xffffffffu, v.x), norm = __reduce_max_sync(0xffffffffu, v.y);
}

// The pre-pass of a (sequence, group) that a block, or a cluster of `cluster` blocks, holds in registers, CHUNKS float4 a thread: it reads the
// group's rows once, all loads under way together, knows the maxima after one barrier and writes the planes out of registers.
// `blk`: the block's, or its cluster's, place among the launch's.
template <int LP, int NC, int CHUNKS>
__device__ __forceinline__ void pass_held(const PassArgs &a, int blk, int rank, int cluster) {
    constexpr int NG = kOneThreads / LP, U = CHUNKS / NC;
    __shared__ uint32_t red[2][kOneThreads / 32];
    const PassUnit w = pass_locate(a, a.n, blk);
    const PassTensor &t = a.t[w.z];
    const int gi = threadIdx.x / LP, li = threadIdx.x % LP;
    const long long plane = (long long)t.batch * t.rows * t.heads * a.pd;
    const int n4 = a.dim >> 2;
    // this lane group's units, as places beyond the (sequence, group)'s first; -1: none
    const long long first = (long long)w.b * t.rows * t.heads + w.g * t.group;
    int place[U];
    {
        int r = (rank * NG * U + gi) / t.group, i = rank * NG * U + gi - r * t.group;
        const int dr = NG / t.group, di = NG - dr * t.group;
#pragma unroll
        for (int k = 0; k < U; ++k) {
            place[k] = r < t.rows ? r * t.heads + i : -1;
            r += dr, i += di;
            if (i >= t.group) i -= t.group, ++r;
        }
    }
    float4 x[U][NC];
#pragma unroll
    for (int k = 0; k < U; ++k)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int ch = li + LP * c;
            x[k][c] = place[k] >= 0 && ch < n4 ? reinterpret_cast<const float4 *>(t.x + (first + place[k]) * a.dim)[ch] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    float amax = 0.f, nmax = 0.f;
#pragma unroll
    for (int k = 0; k < U; ++k) {
        float sq = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const float4 v = x[k][c];
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
            sq = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, sq))));
        }
        if (!t.nmax) continue;
#pragma unroll
        for (int off = LP / 2; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
        nmax = fmaxf(nmax, sqrtf(sq));
    }
    // (f32 bit patterns of non-negative numbers order like integers)
    const uint32_t wa = __reduce_max_sync(0xffffffffu, __float_as_uint(amax)), wn = __reduce_max_sync(0xffffffffu, __float_as_uint(nmax));
    if ((threadIdx.x & 31) == 0) red[0][threadIdx.x >> 5] = wa, red[1][threadIdx.x >> 5] = wn;
    __syncthreads();
    uint32_t top = __reduce_max_sync(0xffffffffu, red[0][threadIdx.x & (kOneThreads / 32 - 1)]);
    uint32_t dn = __reduce_max_sync(0xffffffffu, red[1][threadIdx.x & (kOneThreads / 32 - 1)]);
    if (cluster > 1) cluster_tops(t.part + (long long)w.bg * cluster, rank, cluster, top, dn);
    if (threadIdx.x == 0 && rank == 0) {
        t.amax[w.bg] = top;
        if (t.nmax) t.nmax[w.bg] = dn;
        if (t.clear) t.clear[w.bg] = 0u;
    }
    const float m = block_mult(top);
#pragma unroll
    for (int k = 0; k < U; ++k) {
        const long long at = first + place[k];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int col = (li + LP * c) * 4;
            if (place[k] >= 0 && col < a.pd) store_split4(t.planes + at * a.pd + col, plane, x[k][c], m);
        }
    }
}

// Both launches in one, for forwards whose every (sequence, group) fits the registers of a block, 16 float4 a thread: a launch less in a chain
// that is nothing but launches.  Us, forward of one sequence of 256, 16/16 heads of 64 20.7 -> 15.8, of 12 of 128, 8/8 heads of
// 192 34.1 -> 20.6, forward and backward of one of 256, 4/2 heads of 32 44.1 -> 41.8.
// Two forms: of 16 float4 a thread, and of 4, with three blocks an SM: forward and backward of 7 sequences of 87, 16/16 heads of 32,
// took 38.8 in two launches, 41.6 with the former alone, 36.3 with the latter.
template <int LP, int NC, int CHUNKS>
__global__ void __launch_bounds__(kOneThreads, CHUNKS == kOneFew ? 3 : 1) pass_one_kernel(const __grid_constant__ PassArgs a) {
    pdl_wait();
    pdl_launch();
    pass_held<LP, NC, CHUNKS>(a, (int)blockIdx.x, 0, 1);
}

// The planes without a first launch, where a cluster of up to eight blocks holds a (sequence, group)'s rows: k's and v's beyond what
// pass_one_kernel takes.  Us a forward, two launches -> a cluster a group: one of T 150, 8/2 heads of 128 17.5 -> 12.6; of 700, 32/8 of
// 128 41.3 -> 33.3; of 2048, 8/2 of 64 52.1 -> 46.1; 2 of 400, 12/4 of 32 23.6 -> 17.6; 8 of 512, 32/8 of 64 67.8 -> 59.2; 16 of 1024,
// 16/16 of 64 219 -> 198; 8 of 1024, 32/8 of 256 no change; by single blocks, 64 of 64, 16/4 of 64 40.5 -> 34.9.  (Sixteen blocks a
// cluster: one of 4096, 32/8 of 128 319 -> 325.)
template <int LP, int NC, int HELD>
__global__ void __launch_bounds__(kOneThreads, HELD == kOneFew ? 3 : 1) pass_planes_kernel(const __grid_constant__ PassArgs a) {
    pdl_wait();
    pdl_launch();
    const int at = (int)blockIdx.x / a.cluster;
    pass_held<LP, NC, HELD>(a, at, (int)blockIdx.x - at * a.cluster, a.cluster);
}

// ---- the one launch of a small backward whose k and v were kept -------------------------------------------
// dout's statistics and planes, q's row-scaled planes and the zeros.  A (sequence, group) is a cluster's, of at most eight blocks, which holds its
// rows of dout in shared memory: they are read once, all copies under way together, beside the zeros; out passes by; the maxima are put
// together behind a cluster's barrier; then the planes leave and q, fetched ahead, follows.  Bound by latency: a launch less in the
// chain.  Us, forward and backward, two launches -> this: one of T 256, 4/2 heads of 32 51 -> 45; 4 of 256, 16/16 of 64 55 -> 44.6; 4 of 100,
// 4/2 of 32 32 -> 29.5; 64 of 100, 8/2 of 64 82.6 -> 78.8; 16 of 512, 16/16 of 64 269 -> 263; 16 of 300, 32/8 of 32 205 -> 203.
// Where a group is more than 160 KB its phases, one after the other, take longer than two launches do: one of 1000, 32/8 of 64 105 -> 111,
// 8 of 512 207 -> 209; and so for wider heads: one of 150, 8/2 of 128 67 -> 68, 8 of 256, 32/8 of 128 182 -> 191.
constexpr int kBackThreads = 512, kBackSteps = 20;  // 8 KB of dout a step
template <int LP>
__global__ void __launch_bounds__(kBackThreads, 2) pass_backward_kernel(const __grid_constant__ PassArgs a) {
    constexpr int NG = kBackThreads / LP, S = kPassUnroll;
    extern __shared__ __align__(16) float4 held[];  // [a.per][kBackThreads], a thread's own; then [a.per][NG] norms
    __shared__ uint32_t red[2][kBackThreads / 32];
    pdl_wait();
    pdl_launch();
    const PassTensor &t = a.t[0], &tq = a.t[1];
    const int bg = (int)blockIdx.x / a.cluster, rank = (int)blockIdx.x - bg * a.cluster;
    const int groups = t.heads / t.group, b = bg / groups, g = bg - b * groups, units = t.rows * t.group;
    const int gi = threadIdx.x / LP, li = threadIdx.x % LP, n4 = a.dim >> 2;
    const long long first = (long long)b * t.rows * t.heads + g * t.group, plane = (long long)t.batch * t.rows * t.heads * a.pd;
    float *norms = reinterpret_cast<float *>(held + a.per * kBackThreads) + gi;
    const uint32_t slot0 = (uint32_t)__cvta_generic_to_shared(held + threadIdx.x);
    const int u0 = rank * a.per * NG + gi;
    const auto place = [&](int k) -> long long {  // of the block's k-th unit of this lane group; -1: none
        const int u = u0 + k * NG;
        return k < a.per && u < units ? first + pass_row(t, u) * (t.heads - t.group) + u : -1;
    };
    for (int k = 0; k < a.per; ++k) {
        const long long at = place(k);
        const bool in = at >= 0 && li < n4;
        copy16_async(slot0 + (uint32_t)(k * kBackThreads * 16), reinterpret_cast<const float4 *>(t.x) + (in ? at * n4 + li : 0), in);
    }
    copy_async_commit();
    const auto load = [&](const float *x, int k0, float4 (&r)[S]) {
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const long long at = place(k0 + s);
            r[s] = at >= 0 && li < n4 ? reinterpret_cast<const float4 *>(x)[at * n4 + li] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    float4 r[S];
    load(t.o, 0, r);
    for (int f = 0; f < a.n_fill; ++f) {  // this block's share of the zeros
        const long long n = (a.fill_n4[f] + gridDim.x - 1) / gridDim.x, i0 = n * blockIdx.x, i1 = i0 + n < a.fill_n4[f] ? i0 + n : a.fill_n4[f];
        for (long long i = i0 + threadIdx.x; i < i1; i += kBackThreads) a.fill[f][i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    copy_async_wait<0>();
    float amax = 0.f, nmax = 0.f;
    for (int k0 = 0; k0 < a.per; k0 += S) {
        float sq[S], de[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            sq[s] = de[s] = 0.f;
            if (k0 + s >= a.per) continue;
            const float4 x = held[(k0 + s) * kBackThreads + threadIdx.x], o = r[s];
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));
            sq[s] = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w)));
            de[s] = fmaf(x.x, o.x, fmaf(x.y, o.y, fmaf(x.z, o.z, x.w * o.w)));
        }
        if (k0 + S < a.per) load(t.o, k0 + S, r);
        else load(tq.x, 0, r);  // (q's first rows, for behind the barrier)
#pragma unroll
        for (int s = 0; s < S; ++s) {
#pragma unroll
            for (int off = LP / 2; off > 0; off >>= 1) {
                sq[s] += __shfl_xor_sync(0xffffffffu, sq[s], off);
                de[s] += __shfl_xor_sync(0xffffffffu, de[s], off);
            }
            const float norm = sqrtf(sq[s]);
            nmax = fmaxf(nmax, norm);
            const long long at = place(k0 + s);
            if (li == 0 && at >= 0) t.delta[at] = de[s], t.rnorm[at] = norm, norms[(k0 + s) * NG] = norm;
        }
    }
    // (f32 bit patterns of non-negative numbers order like integers)
    const uint32_t wa = __reduce_max_sync(0xffffffffu, __float_as_uint(amax)), wn = __reduce_max_sync(0xffffffffu, __float_as_uint(nmax));
    if ((threadIdx.x & 31) == 0) red[0][threadIdx.x >> 5] = wa, red[1][threadIdx.x >> 5] = wn;
    __syncthreads();
    uint32_t top = __reduce_max_sync(0xffffffffu, red[0][threadIdx.x & (kBackThreads / 32 - 1)]);
    uint32_t dn = __reduce_max_sync(0xffffffffu, red[1][threadIdx.x & (kBackThreads / 32 - 1)]);
    if (a.cluster > 1) cluster_tops(t.part + (long long)bg * a.cluster, rank, a.cluster, top, dn);
    if (threadIdx.x == 0 && rank == 0) t.amax[bg] = top, t.nmax[bg] = dn;
    const float m = block_mult(top), mq = block_mult(tq.amax[bg]);
    const uint32_t vn = tq.vn_final[bg];
    const bool in_planes = li * 4 < a.pd;
    for (int k = 0; k < a.per; ++k) {
        const long long at = place(k);
        if (at >= 0 && in_planes) store_split4(t.planes + at * a.pd + li * 4, plane, held[k * kBackThreads + threadIdx.x], m);
    }
    for (int k0 = 0; k0 < a.per; k0 += S) {
        float4 x[S];
#pragma unroll
        for (int s = 0; s < S; ++s) x[s] = r[s];
        if (k0 + S < a.per) load(tq.x, k0 + S, r);
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const long long at = place(k0 + s);
            if (at < 0 || !in_planes) continue;
            float cq, rel;
            ds_row_scale(norms[(k0 + s) * NG], dn, vn, cq, rel);
            store_split4(tq.qs + at * a.pd + li * 4, plane, x[s], mq * rel);
        }
    }
}

// ---- host side --------------------------------------------------------------------------------------
// Slots of one tensor of `bg` (sequence, group) pairs: what pass_slots() below can ask for.
inline size_t pass_part_bytes(size_t bg) { return (bg > (size_t)kPassTargetBlocks ? bg : (size_t)kPassTargetBlocks) * sizeof(uint2); }

// Adds a tensor to the launch.
inline PassTensor &pass_add(PassArgs &a, const float *x, int batch, int rows, int heads, int group, uint2 *part, uint32_t *amax,
                            uint32_t *nmax, __half *planes) {
    PassTensor &t = a.t[a.n++];
    t = PassTensor{};
    t.x = x, t.batch = batch, t.rows = rows, t.heads = heads, t.group = group;
    t.part = part, t.amax = amax, t.nmax = nmax, t.planes = planes;
    // (exact up to u with u times what the rounding up added, less than group, below 2^32; the last block's lanes look a step further)
    if (group > 1 && ((unsigned long long)rows * group + (1u << 20)) * (unsigned)group < (1ull << 32)) t.per_head = (uint32_t)(((1ull << 32) + group - 1) / group);
    const long long bg = (long long)batch * (heads / group), units = (long long)rows * group;
    // 2048 blocks a tensor, 14 an SM (4096 and 1024 were 1-2 % slower, 512 more), of at least 256 units at 32 columns, 128 up
    // to 64 and 64 beyond: eight units a lane group where 32 lanes hold one, two at 80 and 96 columns and four at 192, whose
    // units are held by 8 and 16 lanes.  Eight there too is 1-2 % of a large step faster (8 sequences of 512, 16/4 heads of 96,
    // 223 -> 220 us) and costs a small one up to a quarter (one of 500, 8/2 heads of 80, 69 -> 87).
    const int lanes = a.dim <= 32 ? 8 : (a.dim <= 64 ? 16 : 32);
    const long long step = (long long)kPassThreads / lanes * 8;
    long long slots = kPassTargetBlocks / bg;
    slots = slots > kPassMaxSlots ? kPassMaxSlots : (slots < 1 ? 1 : slots);
    const long long most = (units + step - 1) / step;
    if (slots > most) slots = most;
    t.slots = (int)slots;
    return t;
}
inline void pass_fill(PassArgs &a, float *dst, long long n) {
    a.fill[a.n_fill] = reinterpret_cast<float4 *>(dst), a.fill_n4[a.n_fill++] = n / 4;
}
// The blocks that a (sequence, group) of the one-launch forms needs at `units` units each; 0: the forms do not take the call, because a tensor
// is rotated, or more than planes and maxima are wanted, or the tensors need different numbers of blocks.  A cluster has as many for one
// tensor as for the other, so that some would have no unit, and no launch has such blocks: twice in some twenty runs of a suite of
// calls an illegal address ended one of two projections whose clusters had them (the maxima met in distributed shared memory then).  No
// cause has been found, in those blocks or elsewhere.
inline long long pass_one_blocks(const PassArgs &a, int units) {
    long long need = 0;
    for (int i = 0; i < a.n; ++i) {
        const PassTensor &t = a.t[i];
        if (!t.part || t.delta || t.rope || t.qs) return 0;
        const long long blocks = ((long long)t.rows * t.group + units - 1) / units;
        if (need && blocks != need) return 0;
        need = blocks;
    }
    return a.n_fill == 0 ? need : 0;
}
// Whether pass_one_kernel does.  (Its line is still the one drawn when the launch converted the query rows as well, which count although the
// forward reads those itself, and so is pass_one_pays: beyond them the forms of pass_planes_kernel take over.)
inline bool pass_takes_one(const PassArgs &a, int units) { return a.q_units <= units && pass_one_blocks(a, units) == 1; }
inline int pass_sm_count() {
    const DeviceInfo *d = device_info();
    return d && d->sm_count > 0 ? d->sm_count : 148;
}
// Whether it pays in the form of 16 float4 a thread, where a block has an SM to itself however few units its (sequence, group) has: a wave
// takes 4.5 us almost empty and 7 full, and what the two launches take goes with the bytes, so the emptier the blocks the fewer waves pay; with
// groups of query heads k's and v's blocks are the empty ones, without them the two launches have small blocks as well.  Us, forward's
// pre-pass in two launches / one, by the room in use and the waves: 16/4 heads of 64, T 48 (0.19) 3.9 waves 24 / 23.4, 5.2 27.5 / 31, 20.8
// 70 / 95; T 64 (0.25) 3.9 27 / 25, 10.4 46 / 55; T 80 (0.31) 5.2 38 / 33, 10.4 58 / 58, 20.8 96 / 103; T 100 (0.39) 10.4 69 / 62, 20.8
// 112 / 109; 16/16 heads of 40, T 130 (0.25) 15.6 79 / 77, 41.5 156 / 186; of 64, T 160 (0.31) 20.8 109 / 102, 41.5 177 / 196; of 96, T 70
// (0.22) 20.8 104 / 78, 41.5 145 / 149; from two fifths on one launch was the faster for any number of waves.
inline bool pass_one_pays(const PassArgs &a, int units, int sms) {
    const long long bg = (long long)a.t[0].batch * (a.t[0].heads / a.t[0].group);
    long long blocks = a.q_units ? bg : 0, held = bg * a.q_units;
    bool groups = a.q_units > a.t[0].rows;
    for (int i = 0; i < a.n; ++i) {
        const PassTensor &t = a.t[i];
        blocks += (long long)t.batch * (t.heads / t.group), held += (long long)t.batch * t.rows * t.heads;
        groups |= t.group > 1;
    }
    const double in_use = (double)held / ((double)blocks * units), waves = (double)blocks / sms;
    return in_use >= 0.4 || waves <= (groups ? 80. : 450.) * in_use * in_use;
}
// The same of pass_planes_kernel's form of 16, for k and v alone (a cluster's blocks are two thirds full at least; a single block, which comes
// here where two or more of 4 float4 would have too few slots, may be almost empty).  Us a forward, two launches / one, 16/16 heads, by the
// room in use: of 64, 128 sequences, 0.25 217 / 270, 0.39 279 / 309, 0.50 314 / 332, 0.59 417 / 424, 0.78 589 / 566, 1 676 / 633; of 32, 0.50 528 /
// 537, 0.68 833 / 810; of 128, 64 sequences, 0.39 136 / 149, 0.50 149 / 161, 0.70 239 / 235; where a unit is two or three chunks a
// lane, earlier: of 96, 0.31 131 / 123; of 192, 0.25 115 / 123, 0.41 161 / 145; of 256, 0.31 134 / 142, 0.47 159 / 155.
// (Few blocks: a launch less is all that counts.)
inline bool pass_held_pays(const PassArgs &a, int units, long long cluster, int chunks, int sms) {
    long long blocks = 0, held = 0;
    for (int i = 0; i < a.n; ++i) {
        const PassTensor &t = a.t[i];
        blocks += (long long)t.batch * (t.heads / t.group) * cluster, held += (long long)t.batch * t.rows * t.heads;
    }
    return blocks <= sms || (double)held >= (chunks == 1 ? 0.64 : 0.4) * blocks * units;
}
// Blocks that hold their (sequence, group)s' rows, `cluster` of them one.
template <typename Kernel>
inline int launch_pass_held(const char *name, Kernel kernel, PassArgs &a, int cluster, cudaStream_t stream) {
    long long blocks = 0;
    a.cluster = cluster;
    for (int i = 0; i < a.n; ++i) {
        PassTensor &t = a.t[i];
        t.slots = 1, t.first = (int)blocks;
        blocks += (long long)t.batch * (t.heads / t.group);
    }
    if (blocks * cluster > 0x7fffffffLL) return refuse("the operand planes of this shape need more blocks than a launch can have.");
    const dim3 grid((unsigned)(blocks * cluster)), th(kOneThreads);
    return cluster > 1 ? launch_pdl_cluster(name, kernel, grid, th, 0, stream, cluster, a) : launch_pdl(name, kernel, grid, th, 0, stream, a);
}
// Blocks of a (sequence, group) of `steps` steps in a backward's one launch, and the steps that each takes: eight steps a block, or as many blocks as
// give every SM one.  Every block has a step.
struct PassBackPlan {
    int cluster, per;
};
inline PassBackPlan pass_backward_plan(long long steps, long long bg, int sms) {
    long long c = (steps + 7) / 8;
    const long long fill = (sms + bg - 1) / bg;
    if (c < fill) c = fill;
    if (c > steps) c = steps;
    if (c > kOneCluster) c = kOneCluster;
    const long long per = (steps + c - 1) / c;
    return PassBackPlan{(int)((steps + per - 1) / per), (int)per};
}
// The one launch of a backward (dout in a.t[0], q in a.t[1]); -1: not taken, because more is wanted, the rows are too many or too wide, or out
// starts on a 4-byte boundary.
inline int launch_pass_backward_one(PassArgs &a, cudaStream_t stream) {
    const PassTensor &t = a.t[0], &q = a.t[1];
    if (a.n != 2 || a.pd > 64 || q.part || !q.qs || q.rope || !t.part || !t.delta || !t.nmax || (reinterpret_cast<uintptr_t>(t.o) & 15u) != 0) return -1;
    const int ng = kBackThreads / (a.pd <= 32 ? 8 : 16);
    const long long bg = (long long)t.batch * (t.heads / t.group), steps = ((long long)t.rows * t.group + ng - 1) / ng;
    if (steps > kBackSteps) return -1;
    const PassBackPlan plan = pass_backward_plan(steps, bg, pass_sm_count());
    if (plan.cluster > 1 && bg * plan.cluster > kPassTargetBlocks) return -1;  // (the slots that dout has)
    const int c = a.cluster = plan.cluster;
    a.per = plan.per;
    const size_t smem = (size_t)a.per * (kBackThreads * sizeof(float4) + ng * sizeof(float));
    const auto kernel = a.pd <= 32 ? pass_backward_kernel<8> : pass_backward_kernel<16>;
    if (optin_smem((const void *)kernel, smem)) return 1;
    const dim3 grid((unsigned)(bg * c)), th(kBackThreads);
    return c > 1 ? launch_pdl_cluster("pass_backward_kernel", kernel, grid, th, smem, stream, c, a) : launch_pdl("pass_backward_kernel", kernel, grid, th, smem, stream, a);
}
// Both launches (or the second alone, for zeros).  The tensors whose maxima are wanted come first in a.t.
inline int launch_pass(PassArgs &a, cudaStream_t stream) {
    long long blocks = 0, stats = 0;
    bool o4 = false;
    a.n_stats = 0;
    for (int i = 0; i < a.n; ++i) {
        PassTensor &t = a.t[i];
        t.first = (int)blocks;
        blocks += (long long)t.batch * (t.heads / t.group) * t.slots;
        if (t.part) a.n_stats = i + 1, stats = blocks;
        o4 |= (reinterpret_cast<uintptr_t>(t.o) & 15u) != 0;
    }
    a.fill_first[0] = (int)blocks;
    for (int f = 0; f < a.n_fill; ++f) {
        blocks += (a.fill_n4[f] + kFillPerBlock - 1) / kFillPerBlock;
        a.fill_first[f + 1] = (int)blocks;
    }
    if (blocks > 0x7fffffffLL) return refuse("the operand planes of this shape need more blocks than a launch can have.");
    int rc;
    const dim3 gs((unsigned)stats), gp((unsigned)blocks), th(kPassThreads);
    // lanes x chunks of four columns that a unit takes: the tightest that holds it
    const auto both = [&](auto lanes, auto chunks) -> int {
        constexpr int LP = lanes.value, NC = chunks.value;
        constexpr int few = pass_one_units<LP, NC, kOneFew>(), most = pass_one_units<LP, NC, kOneMost>();
        if (pass_takes_one(a, few)) return launch_pass_held("pass_one_kernel", pass_one_kernel<LP, NC, kOneFew>, a, 1, stream);
        if (pass_takes_one(a, most) && pass_one_pays(a, most, pass_sm_count())) return launch_pass_held("pass_one_kernel", pass_one_kernel<LP, NC, kOneMost>, a, 1, stream);
        // (every block of a cluster has a slot of its tensor's)
        long long bg = 0;
        for (int i = 0; i < a.n; ++i) bg = std::max(bg, (long long)a.t[i].batch * (a.t[i].heads / a.t[i].group));
        const auto fits = [&](long long c) { return c > 0 && c <= kOneCluster && bg * c <= kPassTargetBlocks; };
        long long c = pass_one_blocks(a, few);
        if (fits(c)) return launch_pass_held("pass_planes_kernel", pass_planes_kernel<LP, NC, kOneFew>, a, (int)c, stream);
        c = pass_one_blocks(a, most);
        if (fits(c) && pass_held_pays(a, most, c, NC, pass_sm_count())) return launch_pass_held("pass_planes_kernel", pass_planes_kernel<LP, NC, kOneMost>, a, (int)c, stream);
        const size_t smem = (size_t)kStatsStages * NC * 2 * kPassThreads * sizeof(float4);
        const auto stats_kernel = o4 ? pass_stats_kernel<LP, NC, true> : pass_stats_kernel<LP, NC, false>;
        if (optin_smem((const void *)stats_kernel, smem)) return 1;
        rc = stats ? launch_pdl("pass_stats_kernel", stats_kernel, gs, th, smem, stream, a) : 0;
        return rc ? rc : launch_pdl("pass_planes_kernel", pass_planes_kernel<LP, NC>, gp, th, 0, stream, a);
    };
    using std::integral_constant;
    if (a.pd <= 32) return both(integral_constant<int, 8>{}, integral_constant<int, 1>{});
    if (a.pd <= 64) return both(integral_constant<int, 16>{}, integral_constant<int, 1>{});
    if (a.pd <= 96) return both(integral_constant<int, 8>{}, integral_constant<int, 3>{});
    if (a.pd <= 128) return both(integral_constant<int, 32>{}, integral_constant<int, 1>{});
    if (a.pd <= 192) return both(integral_constant<int, 16>{}, integral_constant<int, 3>{});
    return both(integral_constant<int, 32>{}, integral_constant<int, 2>{});
}

}  // namespace tcb
}  // namespace zt
