// Launches of the tensor-core kernels that would leave most SMs without a block are split further: the forward along
// the keys a query tile sees, the backward along the walk of a key tile (the heads of its group, then the query tiles).
// Every part writes a partial result of its own into the workspace and a small kernel puts the parts together in a
// fixed order, so results stay reproducible.
// B200, us before -> after: forward of a window of 64 rows at 4000 keys, 8/2 heads of 128, 92 -> 33; 300 rows at 8000
// keys, 12/4 heads of 64, 151 -> 55; 128 rows at 8000 keys, 32/8 heads of 256, 610 -> 225; forward and backward of one
// sequence, 32/8 heads of 128, T 500 175 -> 96, T 1000 323 -> 228; 4/2 heads of 32, T 2000 211 -> 105;
// 4/2 heads of 64, T 8000 813 -> 526 (126 blocks, half of them walking less than half of the longest); batch 4,
// 16/4 heads of 80, T 1000 373 -> 359.
#pragma once

#include "tc_common.cuh"
#include "zt_common.cuh"

namespace zt {

inline int split_sm_count() {
    const DeviceInfo *d = device_info();
    return d && d->sm_count > 0 ? d->sm_count : 148;  // (no device: a size query; a B200's count stands in)
}

// The order in which the blocks of a launch start (x fastest, then y, then z), where their walks differ in length.  Sequence by
// sequence, blocks that run together share a sequence's operands in L2, which is worth 10 % of the backward at batch 8, T 4096;
// but the last sequence's longest walks then start when the launch is nearly over, and with few blocks an SM that is what
// the launch waits for: at batch 8, T 512, 32/8 heads of 64 the busiest SM of the backward had 1.6 times the average's work.
// So launches of a few blocks an SM go tile by tile through all sequences, longest walks first: up to four in the backward, two
// in the forward.  Us, by sequence -> by tile (blocks):
//   backward  batch 8, T 512, 32/8 heads of 64 174 -> 139 (256), of 128 235 -> 194 (256); batch 4, T 1000, 16/4 heads of 80
//             178 -> 127 (256, walks split); batch 8, T 768, of 128 393 -> 366 (384), T 1024 620 -> 602 (512), T 1536 no
//             difference (768), T 2048 4 % slower (1024)
//   forward   two heads a block: batch 4, T 1024, 16/4 heads of 128 72 -> 59 (256); batch 8, T 512, 32/8, with its
//             pre-pass 149 -> 158 (512).  One head a block: batch 16, T 512, 12/4 heads 93 -> 103 (768).  Wide heads: batch
//             2, T 1024, 16/4 heads of 256 102 -> 76 (256)
// (One wave starts together, in whatever order.)
constexpr int kFwdTileWaves = 2, kBwdTileWaves = 4;
inline bool tile_by_tile(long long blocks, int waves) {
    return blocks > split_sm_count() && blocks <= (long long)waves * split_sm_count();
}
// The grid for `across` blocks (heads, head pairs, KV heads) of each of `tiles` tiles of each of `seqs` sequences (times the
// parts that a walk is split into): the sequences along z, or behind each other along x.
inline dim3 tile_major_grid(int across, int tiles, int seqs, int waves) {
    return tile_by_tile((long long)across * tiles * seqs, waves) ? dim3((unsigned)(across * seqs), (unsigned)tiles)
                                                                 : dim3((unsigned)across, (unsigned)tiles, (unsigned)seqs);
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

// Parts of the backward's walk: heads x ranges of query tiles.  A step is a query tile of bwd_step_rows rows of one head.  (Of one
// tile, where all there are is 64 rows at 64 columns.)
constexpr int bwd_step_rows(int dim) { return dim <= 64 ? 128 : 64; }
struct BwdParts {
    int heads, ranges;
    __host__ __device__ int n() const { return heads * ranges; }
};
// The split with the shortest schedule, in steps (about 3 us each, 64 rows at 128 columns or 128 at 64): a launch ends with
// its longest block, or once all blocks' steps have been shared out with half a block left over at the end (the walks are of
// all lengths, longest first); a block costs three steps beside its walk (two at 64 columns, whose tiles are half as large),
// putting the parts together two and their traffic one per 45 blocks (at 64 columns, whose parts are half as large,
// one and a half and one per 90).  Parts keep 256 rows of the longest walk, and a launch two blocks an SM (which bounds the
// partial results: 38 MB at most).  At 64 columns, us a step unsplit / split as this does (heads x ranges): batch 4, T 1000, 16/4
// heads 210 / 180 (2 x 1); one sequence, 32/8 heads, T 1000 180 / 122 (4 x 1), T 2048 332 / 246 (2 x 1); 8/2 heads, T 512 87 / 53 (4 x 2).
inline BwdParts bwd_parts(int batch, int T, int n_heads, int n_kv_heads, int dim) {
    const int rows = bwd_step_rows(dim), group = n_heads / n_kv_heads, tiles = (T + rows - 1) / rows, sms = split_sm_count();
    const long long key_tiles = (T + 127) / 128, ctas = n_kv_heads * key_tiles * batch;
    const double walks = (double)group * (tiles * key_tiles - key_tiles * (key_tiles - 1) / 2 * (128 / rows)) * n_kv_heads * batch;  // all blocks' steps
    const bool narrow = rows == 128;
    const double block = narrow ? 2 : 3, join = narrow ? 1.5 : 2, traffic = narrow ? 90 : 45;
    BwdParts best{1, 1};
    if (ctas > 2 * sms) return best;
    double best_cost = 0.;
    for (int h = 1; h <= group; ++h) {
        if (group % h != 0) continue;
        for (int r = 1; r == 1 || r * 128 <= tiles * rows; ++r) {
            const int n = h * r;
            if (n > 1 && (n * ctas > 2 * sms || (long long)group * tiles * rows < 256LL * n)) break;
            const double longest = (double)(group / h) * ((tiles + r - 1) / r) + 3, shared = (walks + block * n * ctas) / sms + longest / 2;
            double cost = n * ctas <= sms || longest > shared ? longest : shared;
            if (n > 1) cost += join + n * ctas / traffic;
            // (of equals the split by heads: a part of a range also flushes its accumulators once per head)
            if ((h == 1 && r == 1) || cost <= best_cost) best = BwdParts{h, r}, best_cost = cost;
        }
    }
    return best;
}
inline size_t bwd_parts_floats(int batch, int T, int n_heads, int n_kv_heads, int dim) {
    const int n = bwd_parts(batch, T, n_heads, n_kv_heads, dim).n();
    return n < 2 ? 0 : (size_t)n * 2 * batch * T * n_kv_heads * dim;
}

// Neither number grows with the shape -- a shorter sequence may be split where a longer one is not -- so a scratch that is to
// serve every smaller shape too takes these, which do: the blocks that a split ends at, times what one of them writes.
inline size_t fwd_parts_floats_bound(int dim) { return (size_t)split_sm_count() * 128 * (2 * (size_t)dim + 1); }
inline size_t bwd_parts_floats_bound(int batch, int T, int n_heads, int dim) {
    const size_t by_blocks = (size_t)4 * split_sm_count() * 128 * dim;
    const int rows = bwd_step_rows(dim);
    const size_t by_steps = (size_t)n_heads * ((T + rows - 1) / rows) * rows / 256 * 2 * batch * T * dim;  // (a part keeps 256 rows of whole steps)
    return by_steps < by_blocks ? by_steps : by_blocks;
}

// out, lse <- the forward's parts.  A warp per (row, head).
__global__ void __launch_bounds__(256) fwd_join_kernel(const float *part, const float *part_lse, float *out, float *lse, long long rows,
                                                       int dim, int parts) {
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
__global__ void __launch_bounds__(256) bwd_join_kernel(const float *part, float *dk, float *dv, int batch, int T, int width,
                                                       BwdParts parts, int rows) {
    pdl_wait();
    pdl_launch();
    const long long n4 = (long long)batch * T * width / 4;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n4) return;
    const int t = (int)(i * 4 / width % T);
    const int per_head = (T + rows - 1) / rows - t / 128 * (128 / rows), per = (per_head + parts.ranges - 1) / parts.ranges;
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
inline int launch_bwd_join(const float *part, float *dk, float *dv, int batch, int T, int width, BwdParts parts, int rows, cudaStream_t stream) {
    const long long n4 = (long long)batch * T * width / 4;
    return launch_pdl("bwd_join_kernel", bwd_join_kernel, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, stream, part, dk, dv, batch, T,
                      width, parts, rows);
}

}  // namespace zt
