// Launches of the tensor-core kernels that would leave most SMs without a block are split further: the forward along
// the keys a query tile sees, the backward along the walk of a key tile (the heads of its group, then the query tiles).
// Every part writes a partial result of its own into the workspace and a small kernel puts the parts together in a
// fixed order, so results stay reproducible.
// B200, us before -> after: forward of a window of 64 rows at 4000 keys, 8/2 heads of 128, 92 -> 33; 300 rows at 8000
// keys, 12/4 heads of 64, 151 -> 55; 128 rows at 8000 keys, 32/8 heads of 256, 610 -> 225; forward and backward of one
// sequence, 32/8 heads of 128, T 500 175 -> 96, T 1000 323 -> 228; 4/2 heads of 32, T 2000 211 -> 105.
#pragma once

#include "tc_common.cuh"
#include "zt_common.cuh"

namespace zt {

inline int split_sm_count() {
    const DeviceInfo *d = device_info();
    return d && d->sm_count > 0 ? d->sm_count : 148;  // (no device: a size query; a B200's count stands in)
}

// Parts of the forward along the keys.  A part should keep four key tiles of 64: fewer cost more in the part's own
// prologue and in putting the rows together than they save.
inline int fwd_parts(int batch, int T, int n_heads, int q_offset) {
    const long long ctas = (long long)((T + 127) / 128) * n_heads * batch, tiles = ((long long)q_offset + T + 63) / 64;
    if (tiles < 12) return 1;
    long long n = split_sm_count() / ctas;
    if (n > tiles / 4) n = tiles / 4;
    return n < 2 ? 1 : (n > 16 ? 16 : (int)n);
}
// Floats of the forward's partial results: rows of out (twice as many where O is also summed in memory on the way), then
// the log-sum-exp of every row.
inline size_t fwd_parts_floats(int batch, int T, int n_heads, int dim, int q_offset) {
    const int n = fwd_parts(batch, T, n_heads, q_offset);
    const size_t rows = (size_t)batch * T * n_heads;
    return n < 2 ? 0 : n * rows * ((q_offset > 0 ? 2 : 1) * (size_t)dim + 1);
}

// Parts of the backward's walk: heads x ranges of query tiles.  A part keeps four steps (a query tile of 64 rows of one
// head each) of the longest walk.
struct BwdParts {
    int heads, ranges;
    __host__ __device__ int n() const { return heads * ranges; }
};
inline BwdParts bwd_parts(int batch, int T, int n_heads, int n_kv_heads) {
    const long long ctas = (long long)n_kv_heads * ((T + 127) / 128) * batch;
    const int group = n_heads / n_kv_heads, tiles = (T + 63) / 64;
    const long long most = (long long)group * tiles / 4, fit = split_sm_count() / ctas;
    const int want = (int)(fit < most ? fit : most);
    BwdParts p{1, 1};
    if (want < 2) return p;
    for (int h = 1; h <= group && h <= want; ++h)
        if (group % h == 0) p.heads = h;
    p.ranges = want / p.heads < tiles / 2 ? want / p.heads : tiles / 2;
    if (p.ranges < 1) p.ranges = 1;
    return p;
}
inline size_t bwd_parts_floats(int batch, int T, int n_heads, int n_kv_heads, int dim) {
    const int n = bwd_parts(batch, T, n_heads, n_kv_heads).n();
    return n < 2 ? 0 : (size_t)n * 2 * batch * T * n_kv_heads * dim;
}

// out, lse <- the forward's parts.  A warp per (row, head).
__global__ void __launch_bounds__(256) fwd_join_kernel(const float *__restrict__ part, const float *__restrict__ part_lse,
                                                       float *__restrict__ out, float *__restrict__ lse, long long rows, int dim,
                                                       int parts) {
    pdl_wait();
    pdl_launch();
    const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31, n4 = dim >> 2;
    const float mine = lane < parts ? part_lse[lane * rows + row] : -INFINITY;  // (at most 16 parts)
    float top = mine;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
    float w = (mine == -INFINITY) ? 0.f : ex2((mine - top) * kLog2e), sum = w;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    w /= sum;
    for (int c = lane; c - lane < n4; c += 32) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = 0; i < parts; ++i) {
            const float wi = __shfl_sync(0xffffffffu, w, i);
            if (wi == 0.f || c >= n4) continue;
            const float4 x = *(reinterpret_cast<const float4 *>(part + ((long long)i * rows + row) * dim) + c);
            a.x = fmaf(wi, x.x, a.x), a.y = fmaf(wi, x.y, a.y), a.z = fmaf(wi, x.z, a.z), a.w = fmaf(wi, x.w, a.w);
        }
        if (c < n4) *(reinterpret_cast<float4 *>(out + row * dim) + c) = a;
    }
    if (lse && lane == 0) lse[row] = top + log2f(sum) * kLn2;
}
inline int launch_fwd_join(const float *part, const float *part_lse, float *out, float *lse, long long rows, int dim, int parts,
                           cudaStream_t stream) {
    return launch_pdl("fwd_join_kernel", fwd_join_kernel, dim3((unsigned)((rows + 7) / 8)), dim3(256), 0, stream, part, part_lse, out,
                      lse, rows, dim, parts);
}

// dk, dv <- the backward's parts, each [2][batch][T][width] (dk, then dv).  A range of query tiles that lies before the
// key tile wrote nothing.
__global__ void __launch_bounds__(256) bwd_join_kernel(const float *__restrict__ part, float *__restrict__ dk, float *__restrict__ dv,
                                                       int batch, int T, int width, BwdParts parts) {
    pdl_wait();
    pdl_launch();
    const long long n4 = (long long)batch * T * width / 4;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n4) return;
    const int t = (int)(i * 4 / width % T);
    const int per_head = (T + 63) / 64 - t / 128 * 2, per = (per_head + parts.ranges - 1) / parts.ranges;
    const float4 *src = reinterpret_cast<const float4 *>(part);
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    for (int s = 0; s < parts.n(); ++s) {
        if (s % parts.ranges * per >= per_head) continue;
        const float4 x = src[s * 2 * n4 + i], y = src[(s * 2 + 1) * n4 + i];
        a.x += x.x, a.y += x.y, a.z += x.z, a.w += x.w;
        b.x += y.x, b.y += y.y, b.z += y.z, b.w += y.w;
    }
    reinterpret_cast<float4 *>(dk)[i] = a, reinterpret_cast<float4 *>(dv)[i] = b;
}
inline int launch_bwd_join(const float *part, float *dk, float *dv, int batch, int T, int width, BwdParts parts, cudaStream_t stream) {
    const long long n4 = (long long)batch * T * width / 4;
    return launch_pdl("bwd_join_kernel", bwd_join_kernel, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, stream, part, dk, dv, batch, T,
                      width, parts);
}

}  // namespace zt
