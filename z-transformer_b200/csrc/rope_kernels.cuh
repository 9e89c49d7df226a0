// Rotary position embedding on the input side of attention (src/rope.zig:21-55) and its transpose on
// the gradient side (ropeBackward, src/autograd.zig:851-874).
//
// Row r of a [T, heads * head_dim] tensor sits at absolute position pos + r; element i of a head pairs
// with element i + head_dim/2 of the same head; the angle (pos + r) / theta^(2i / head_dim), its cosine
// and sine and both multiply-adds are f64, with one narrowing to f32 -- the reference's arithmetic.
//
// The (cos, sin) pairs depend on (row, i) only, so they are computed once per call -- angle, cosine
// and sine in f64 -- into a table of T x head_dim/2 float2 (kept in both orders) and read by whoever rotates: the pre-pass of
// the tensor-core kernels, which rotates q and k on their way into the f16 operand planes (the rotated
// f32 tensors are never written), or rope_apply_kernel for the CUDA-core path and for the gradients.
// Departure from the reference's arithmetic: the two multiply-adds are f32 (one fused) on f32-rounded
// cosines and sines, not f64 on f64 ones.  The result differs from the reference's by at most a few
// units in the last place of max(|lo|, |hi|) (2e-7 relative), three orders below the parity bar; what
// must be f64 -- the angle, which reaches thousands of radians -- is.  f64 multiply-adds on a 16-byte
// table entry per element made the rotation cost more than the HBM round trip it is there to save.
#pragma once

#include "zt_common.cuh"

#include <initializer_list>

namespace zt {

// table[r * half + i] = table_t[i * rows + r] = (cos, sin) of (pos + r) / theta^(2 i / head_dim)
__global__ void __launch_bounds__(256) rope_table_kernel(float2 *__restrict__ table, float2 *__restrict__ table_t, int rows,
                                                         int half, int pos, double theta) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)rows * half) return;
    const int r = (int)(idx / half), i = (int)(idx - (long long)r * half);
    const double exponent = (double)(2 * i) / (double)(2 * half);
    const double angle = (double)(pos + r) / pow(theta, exponent);
    double s, c;
    sincos(angle, &s, &c);
    const float2 cs = make_float2((float)c, (float)s);
    table[idx] = cs;
    table_t[(long long)i * rows + r] = cs;
}

// One element of a rotated row: `mine` at index w of its head, `other` its partner (w +- half).
// Forward: lo' = lo c - hi s, hi' = hi c + lo s.  Transpose: lo' = lo c + hi s, hi' = hi c - lo s.
__device__ __forceinline__ float rope_elem(float mine, float other, float2 cs, bool upper, bool transpose) {
    const float s = (upper != transpose) ? cs.y : -cs.y;
    return fmaf(mine, cs.x, other * s);
}

// Four elements of a head's lower half and their partners, rotated (or, transposed, rotated back); p and q hold their four (cos, sin) pairs.
__device__ __forceinline__ void rope_chunk(float4 lo, float4 hi, float4 p, float4 q, float4 &lr, float4 &hr, bool transpose = false) {
    lr.x = rope_elem(lo.x, hi.x, make_float2(p.x, p.y), false, transpose), hr.x = rope_elem(hi.x, lo.x, make_float2(p.x, p.y), true, transpose);
    lr.y = rope_elem(lo.y, hi.y, make_float2(p.z, p.w), false, transpose), hr.y = rope_elem(hi.y, lo.y, make_float2(p.z, p.w), true, transpose);
    lr.z = rope_elem(lo.z, hi.z, make_float2(q.x, q.y), false, transpose), hr.z = rope_elem(hi.z, lo.z, make_float2(q.x, q.y), true, transpose);
    lr.w = rope_elem(lo.w, hi.w, make_float2(q.z, q.w), false, transpose), hr.w = rope_elem(hi.w, lo.w, make_float2(q.z, q.w), true, transpose);
}

// out = R x (transpose = 0) or R^T x (transpose = 1) for x [batch][rows][width]; may run in place: a thread
// owns both elements of a pair.  grid over batch * rows * width / 2 pairs.
__global__ void __launch_bounds__(256) rope_apply_kernel(const float *x, float *out, const float2 *__restrict__ table,
                                                         int batch, int rows, int width, int head_dim, int transpose) {
    const int half = head_dim / 2;
    const long long pairs_per_row = width / 2;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)batch * rows * pairs_per_row) return;
    const long long row = idx / pairs_per_row;  // batch * rows + r
    const int pr = (int)(idx - row * pairs_per_row);
    const int r = (int)(row % rows);
    const int head = pr / half, i = pr - head * half;
    const long long lo_at = row * width + (long long)head * head_dim + i;
    const float lo = x[lo_at], hi = x[lo_at + half];
    const float2 cs = __ldg(table + (long long)r * half + i);
    out[lo_at] = rope_elem(lo, hi, cs, false, transpose != 0);
    out[lo_at + half] = rope_elem(hi, lo, cs, true, transpose != 0);
}

// The same by 16 bytes, for heads whose halves are multiples of four, of up to two tensors of the same rows (a call's q and k, or their
// gradients).  A block takes 1024 elements of a row's lower halves and their partners.  Us, both gradients of batch 2, T 2048, 32/8 heads of
// 128 (168 MB read and written, 26 at the copy rate), by single elements, a launch each -> this: 75 -> 28.
struct RopeTensor {
    const float *x;
    float *out;
    int heads, blocks;  // blocks a row
};
__global__ void __launch_bounds__(256) rope_apply4_kernel(const RopeTensor a, const RopeTensor b, const float2 *__restrict__ table, int rows, int half,
                                                          int transpose) {
    const bool second = (int)blockIdx.y >= a.blocks;
    const RopeTensor &t = second ? b : a;
    const int h4 = half >> 2, c = ((int)blockIdx.y - (second ? a.blocks : 0)) * 256 + threadIdx.x, head = c / h4, i = c - head * h4;
    if (head >= t.heads) return;
    const long long at = ((long long)blockIdx.x * t.heads + head) * 2 * h4 + i;
    const float4 lo = reinterpret_cast<const float4 *>(t.x)[at], hi = reinterpret_cast<const float4 *>(t.x)[at + h4];
    const float4 *cs = reinterpret_cast<const float4 *>(table + (long long)(blockIdx.x % rows) * half) + 2 * i;
    float4 lr, hr;
    rope_chunk(lo, hi, __ldg(cs), __ldg(cs + 1), lr, hr, transpose != 0);
    reinterpret_cast<float4 *>(t.out)[at] = lr, reinterpret_cast<float4 *>(t.out)[at + h4] = hr;
}

inline int launch_rope_table(float2 *table, float2 *table_t, int rows, int head_dim, int pos, double theta,
                             cudaStream_t stream) {
    const long long n = (long long)rows * (head_dim / 2);
    return ZT_LAUNCH("rope_table_kernel", stream,
                     (rope_table_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(table, table_t, rows, head_dim / 2, pos, theta)));
}
inline int launch_rope_single(const float *x, float *out, const float2 *table, int batch, int rows, int width, int head_dim,
                              bool transpose, cudaStream_t stream) {
    const long long n = (long long)batch * rows * (width / 2);
    return ZT_LAUNCH("rope_apply_kernel", stream,
                     (rope_apply_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(x, out, table, batch, rows, width,
                                                                                         head_dim, transpose ? 1 : 0)));
}
// q_out = R q and k_out = R k, or R^T; either may run in place.
inline int launch_rope_apply(const float *q, float *q_out, int n_heads, const float *k, float *k_out, int n_kv_heads, const float2 *table, int batch,
                             int rows, int head_dim, bool transpose, cudaStream_t stream) {
    uintptr_t all = reinterpret_cast<uintptr_t>(table);
    for (const float *x : {q, (const float *)q_out, k, (const float *)k_out}) all |= reinterpret_cast<uintptr_t>(x);
    const auto blocks = [&](int heads) { return (int)(((long long)heads * (head_dim / 8) + 255) / 256); };
    if (head_dim % 8 == 0 && (all & 15u) == 0 && blocks(n_heads) + blocks(n_kv_heads) <= 65535) {
        const RopeTensor a{q, q_out, n_heads, blocks(n_heads)}, b{k, k_out, n_kv_heads, blocks(n_kv_heads)};
        return ZT_LAUNCH("rope_apply4_kernel", stream,
                         (rope_apply4_kernel<<<dim3((unsigned)(batch * rows), (unsigned)(a.blocks + b.blocks)), 256, 0, stream>>>(
                             a, b, table, rows, head_dim / 2, transpose ? 1 : 0)));
    }
    return launch_rope_single(q, q_out, table, batch, rows, n_heads * head_dim, head_dim, transpose, stream) ||
           launch_rope_single(k, k_out, table, batch, rows, n_kv_heads * head_dim, head_dim, transpose, stream);
}

}  // namespace zt
