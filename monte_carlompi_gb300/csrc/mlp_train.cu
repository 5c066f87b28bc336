// Training engine of the surrogate network: the kernels of one Adam step of a whole ensemble
// (all members at once) beside its products (mlp_gemm.cu), so a step is a short, fixed sequence
// of launches that a CUDA graph replays: split-K sums, loss, bias gradients, Adam, the batch's
// gather and the step counter, each one launch for all members; the learning rate and step count
// are read from device memory so a captured step can be replayed unchanged.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "../../include/mcw_mlp.h"
#include "pdl.cuh"

namespace mcw {

namespace {

// Sum of `splits` partial products: dst[g][i][j] = sum_s src[s][g][i][j] (fixed order).
__global__ void reduce_splits_kernel(const float *src, long long s_split, long long s_src_g, long long ld_src,
                                     float *dst, long long s_dst_g, long long ld_dst, int splits, int m, int n) {
    const int g = blockIdx.z;
    const long long total = (long long)m * n;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long i = e / n, j = e % n;
        const float *s = src + (size_t)g * s_src_g + (size_t)i * ld_src + j;
        float acc = 0.f;
        for (int q = 0; q < splits; ++q) acc += s[(size_t)q * s_split];
        dst[(size_t)g * s_dst_g + (size_t)i * ld_dst + j] = acc;
    }
}

// Weighted squared error of `groups` outputs: each block takes a strip of 32 columns x
// kLossRows rows in 32 x 32 tiles; loss[g] += sum w_j d^2 / (m n) (one atomic per block);
// the gradient 2 w_j d / (m n) as f32 and bf16 [m, n] and bf16 transposed [n, m]
// (through a shared-memory tile, so both stores are coalesced).
constexpr int kLossRows = 256;

__global__ void loss_grouped_kernel(const float *y, long long ldy, long long s_y, const float *t, long long ldt,
                                    long long s_t, const float *w, int m, int n, float *g32, long long ldg,
                                    long long s_g32, __nv_bfloat16 *g16, long long s_g16, __nv_bfloat16 *g16t,
                                    long long ldgt, long long s_g16t, float *loss) {
    __shared__ __nv_bfloat16 tile[32][33];
    __shared__ float wsum[8];
    const int g = blockIdx.z;
    const int c0 = blockIdx.x * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8 threads
    const float scale = 1.f / ((float)m * (float)n);
    const int c = c0 + tx;
    const float wc = (c < n) ? (w ? w[c] : 1.f) : 0.f;
    float l = 0.f;
    for (int r0 = blockIdx.y * kLossRows; r0 < min(m, (blockIdx.y + 1) * kLossRows); r0 += 32) {
        for (int rr = ty; rr < 32; rr += 8) {
            const int r = r0 + rr;
            __nv_bfloat16 h = __float2bfloat16(0.f);
            if (r < m && c < n) {
                const float d = y[(size_t)g * s_y + (size_t)r * ldy + c] - t[(size_t)g * s_t + (size_t)r * ldt + c];
                l += wc * d * d * scale;
                const float gv = 2.f * wc * d * scale;
                g32[(size_t)g * s_g32 + (size_t)r * ldg + c] = gv;
                h = __float2bfloat16(gv);
                g16[(size_t)g * s_g16 + (size_t)r * ldg + c] = h;
            }
            tile[rr][tx] = h;
        }
        __syncthreads();
        for (int cc = ty; cc < 32; cc += 8) {
            const int cw = c0 + cc, r = r0 + tx;
            if (cw < n && r < m) g16t[(size_t)g * s_g16t + (size_t)cw * ldgt + r] = tile[tx][cc];
        }
        __syncthreads();
    }
    for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (tx == 0) wsum[ty] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) b += wsum[q];
        if (b != 0.f) atomicAdd(loss + g, b);
    }
}

// Bias gradients: out[g * s_out + off_l + j] = sum_i G_l[g][i][j] for the layers of
// the table (fixed summation order: 8 row lanes per column, then the 8 partials).
struct ColsumLayer {
    const float *src;
    long long ld, s_g;
    long long off;     // column 0's offset in out
    int n;
    int pad;
};
struct ColsumTable {
    ColsumLayer l[4];
    int n_layers;
};

// One pass over rows [row0, row1) of every (layer, group): 8 row lanes per column,
// their partial sums combined in a fixed order.  blockIdx.y is the row chunk; the
// result goes to out (one chunk) or to partial[((z * chunks + chunk) * ldp) + col].
__global__ void colsum_grouped_kernel(const ColsumTable tab, int groups, int m, int rows_per_chunk, float *out,
                                      long long s_out, float *partial, int ldp) {
    const int layer = blockIdx.z / groups, g = blockIdx.z % groups;
    const ColsumLayer L = tab.l[layer];
    const int col = blockIdx.x * 32 + (threadIdx.x & 31);
    const int row_lane = threadIdx.x >> 5;
    const int r0 = blockIdx.y * rows_per_chunk, r1 = min(m, r0 + rows_per_chunk);
    __shared__ float part[8][32];
    float acc = 0.f;
    if (col < L.n) {
        const float *s = L.src + (size_t)g * L.s_g + col;
        for (int r = r0 + row_lane; r < r1; r += 8) acc += s[(size_t)r * L.ld];
    }
    part[row_lane][threadIdx.x & 31] = acc;
    __syncthreads();
    if (row_lane == 0 && col < L.n) {
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) t += part[q][threadIdx.x];
        if (partial) partial[((size_t)blockIdx.z * gridDim.y + blockIdx.y) * ldp + col] = t;
        else out[(size_t)g * s_out + L.off + col] = t;
    }
}

// Second pass: the chunks' partial sums added in order.
__global__ void colsum_finish_kernel(const ColsumTable tab, int groups, int chunks, const float *partial, int ldp,
                                     float *out, long long s_out) {
    const int layer = blockIdx.z / groups, g = blockIdx.z % groups;
    const ColsumLayer L = tab.l[layer];
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= L.n) return;
    const float *p = partial + (size_t)blockIdx.z * chunks * ldp + col;
    float t = 0.f;
    for (int c = 0; c < chunks; ++c) t += p[(size_t)c * ldp];
    out[(size_t)g * s_out + L.off + col] = t;
}

// Transposed bf16 copies of weight blocks written by Adam: wt[g * s_t + off_t + c * ld_t + o] = w[o, c] for the block's
// rows o < rows and columns c < cols, which start at offset off in the flat layout.
struct TransposeBlock {
    long long off, off_t, ld_t;
    int rows, cols;
};
struct TransposeTable {
    TransposeBlock b[4];
    int n_blocks;
    int pad;
};

// Adam over the flat parameters of every member (the same update as mcw_mlp_adam),
// lr and the 1-based step count read from device memory; writes the bf16 copy of every
// parameter (w16, the same layout) and the transposed copies of the table's blocks.
__global__ void adam_grouped_kernel(float *w, const float *gr, float *mo, float *ve, __nv_bfloat16 *w16,
                                    long long n, const float *lr_dev, const int *step_dev, float b1, float b2,
                                    float eps, __nv_bfloat16 *wt, long long s_t, const TransposeTable tt) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int g = blockIdx.y;
    if (i >= n) return;
    const int step = *step_dev;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    const float lr = *lr_dev;
    const size_t e = (size_t)g * n + i;
    const float gi = gr[e];
    const float m = b1 * mo[e] + (1.f - b1) * gi;
    const float v = b2 * ve[e] + (1.f - b2) * gi * gi;
    mo[e] = m;
    ve[e] = v;
    const float wn = w[e] - lr * (m / c1) / (sqrtf(v / c2) + eps);
    w[e] = wn;
    const __nv_bfloat16 h = __float2bfloat16(wn);
    w16[e] = h;
    if (wt) {
        for (int q = 0; q < tt.n_blocks; ++q) {
            const TransposeBlock &B = tt.b[q];
            const long long k = i - B.off;
            if (k >= 0 && k < (long long)B.rows * B.cols) {
                const long long o = k / B.cols, c = k % B.cols;
                wt[(size_t)g * s_t + B.off_t + (size_t)c * B.ld_t + o] = h;
            }
        }
    }
}

// The same by tiles, for layouts on 16-byte boundaries (adam_tiled): a block takes 32 rows x 64
// columns of a transposed block, or 2,048 consecutive parameters outside them, eight a thread in
// 16-byte loads and stores; the transposed copy goes through shared memory and leaves in runs of
// 64 bytes (2-byte stores a column apart before).  Bound: 30 bytes a parameter, from L2; five
// members 23 us one parameter a thread, 16 us now.
struct AdamTiles {
    TransposeTable tt;
    int first[5];              // first tile of block q; first[n_blocks]: the rest
    long long seg[6][2];       // the rest: [begin, end) between the blocks
    int seg0[6], n_seg;        // first tile of segment s (after the blocks')
    int tiles;
};

__device__ __forceinline__ void adam8(float *w, const float *gr, float *mo, float *ve, __nv_bfloat16 *w16, size_t e,
                                      float lr, float c1, float c2, float b1, float b2, float eps, uint32_t (&h)[4]) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        float4 wv = reinterpret_cast<float4 *>(w + e)[q], mv = reinterpret_cast<float4 *>(mo + e)[q],
               vv = reinterpret_cast<float4 *>(ve + e)[q];
        const float4 gv = reinterpret_cast<const float4 *>(gr + e)[q];
        float *wp = &wv.x, *mp = &mv.x, *vp = &vv.x;
        const float *gp = &gv.x;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float gi = gp[k];
            const float m = b1 * mp[k] + (1.f - b1) * gi;
            const float v = b2 * vp[k] + (1.f - b2) * gi * gi;
            mp[k] = m;
            vp[k] = v;
            wp[k] = wp[k] - lr * (m / c1) / (sqrtf(v / c2) + eps);
        }
        reinterpret_cast<float4 *>(w + e)[q] = wv;
        reinterpret_cast<float4 *>(mo + e)[q] = mv;
        reinterpret_cast<float4 *>(ve + e)[q] = vv;
        const __nv_bfloat162 lo = __floats2bfloat162_rn(wv.x, wv.y), hi = __floats2bfloat162_rn(wv.z, wv.w);
        h[2 * q] = *reinterpret_cast<const uint32_t *>(&lo);
        h[2 * q + 1] = *reinterpret_cast<const uint32_t *>(&hi);
    }
    *reinterpret_cast<uint4 *>(w16 + e) = make_uint4(h[0], h[1], h[2], h[3]);
}

__global__ void __launch_bounds__(256) adam_tiled_kernel(float *w, const float *gr, float *mo, float *ve,
                                                         __nv_bfloat16 *w16, long long n, const float *lr_dev,
                                                         const int *step_dev, float b1, float b2, float eps,
                                                         __nv_bfloat16 *wt, long long s_t, const AdamTiles at) {
    __shared__ __align__(16) __nv_bfloat16 tile[64][40];     // [column][row], rows of 80 bytes
    __shared__ float corr[2];
    const int g = blockIdx.y, t = blockIdx.x;
    after_previous();
    let_next_start();
    if (threadIdx.x == 0) {
        const int step = *step_dev;
        corr[0] = 1.f - powf(b1, (float)step);
        corr[1] = 1.f - powf(b2, (float)step);
    }
    __syncthreads();
    const float lr = *lr_dev, c1 = corr[0], c2 = corr[1];
    const int nb = at.tt.n_blocks;
    uint32_t h[4];
    if (t >= at.first[nb]) {
        int s = 0;
        while (s + 1 < at.n_seg && t >= at.seg0[s + 1]) ++s;
        const long long i = at.seg[s][0] + (long long)(t - at.seg0[s]) * 2048 + threadIdx.x * 8;
        if (i < at.seg[s][1]) adam8(w, gr, mo, ve, w16, (size_t)g * n + i, lr, c1, c2, b1, b2, eps, h);
        return;
    }
    int q = 0;
    while (q + 1 < nb && t >= at.first[q + 1]) ++q;
    const TransposeBlock &B = at.tt.b[q];
    const int across = (B.cols + 63) / 64;
    const int o0 = (t - at.first[q]) / across * 32, c0 = (t - at.first[q]) % across * 64;
    const int row = threadIdx.x >> 3, c8 = (threadIdx.x & 7) * 8;
    h[0] = h[1] = h[2] = h[3] = 0u;
    if (o0 + row < B.rows && c0 + c8 < B.cols)
        adam8(w, gr, mo, ve, w16, (size_t)g * n + B.off + (size_t)(o0 + row) * B.cols + c0 + c8, lr, c1, c2, b1, b2, eps, h);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        tile[c8 + k][row] = __ushort_as_bfloat16((unsigned short)(h[k >> 1] >> ((k & 1) * 16)));
    __syncthreads();
    const int col = threadIdx.x >> 2, o8 = (threadIdx.x & 3) * 8;
    // (what lies past the block's rows, up to ld_t, is the caller's)
    if (c0 + col < B.cols && o0 + o8 < B.rows) {
        __nv_bfloat16 *dst = wt + (size_t)g * s_t + B.off_t + (size_t)(c0 + col) * B.ld_t + o0 + o8;
        if (o0 + o8 + 8 <= B.rows) {
            *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(&tile[col][o8]);
        } else {
            for (int k = 0; o0 + o8 + k < B.rows; ++k) dst[k] = tile[col][o8 + k];
        }
    }
}

// Batch of the step: rows perm[g][b * batch + i] of the encoded inputs (bf16, row
// pitch 16, as x [batch, 16] and transposed [16, batch]) and of the targets, b the
// step's batch counter (device memory).
__global__ void gather_kernel(const __nv_bfloat16 *x_all, const float *t_all, long long ldt_all, int n_out,
                              const int *perm, long long n_rows, const int *counter, int batch,
                              __nv_bfloat16 *x, long long s_x, __nv_bfloat16 *xt, long long s_xt, float *t,
                              long long ldt, long long s_t, float *loss) {
    const int g = blockIdx.y;
    const int i = blockIdx.x;             // row of the batch
    after_previous();
    let_next_start();
    if (loss && i == 0 && threadIdx.x == 0) loss[g] = 0.f;
    const long long idx = (long long)(*counter) * batch + i;
    if (idx >= n_rows) return;            // more steps than the epoch's batches: nothing to gather
    const long long src = perm[(size_t)g * n_rows + (size_t)idx];
    for (int j = threadIdx.x; j < n_out; j += blockDim.x)
        t[(size_t)g * s_t + (size_t)i * ldt + j] = t_all[(size_t)src * ldt_all + j];
    if (threadIdx.x < 16) {
        const __nv_bfloat16 v = x_all[(size_t)src * 16 + threadIdx.x];
        x[(size_t)g * s_x + (size_t)i * 16 + threadIdx.x] = v;
        if (xt) xt[(size_t)g * s_xt + (size_t)threadIdx.x * batch + i] = v;
    }
}

__global__ void advance_kernel(int *counter, int *step) {
    after_previous();
    let_next_start();
    if (threadIdx.x == 0) {
        *counter += 1;
        *step += 1;
    }
}

// The tiles of a layout whose blocks lie in ascending order on 16-byte boundaries; false otherwise.
bool make_adam_tiles(const TransposeTable &tt, long long n, long long s_t, AdamTiles *out) {
    AdamTiles a;
    memset(&a, 0, sizeof(a));
    a.tt = tt;
    long long at = 0;
    int tiles = 0;
    for (int q = 0; q < tt.n_blocks; ++q) {
        const TransposeBlock &b = tt.b[q];
        if ((b.off & 7) || (b.off_t & 7) || (b.ld_t & 7) || (b.cols & 7) || b.off < at)
            return false;
        a.first[q] = tiles;
        tiles += (b.rows + 31) / 32 * ((b.cols + 63) / 64);
        at = b.off + (long long)b.rows * b.cols;
        at = (at + 7) / 8 * 8;
    }
    if ((n & 7) || (s_t & 7)) return false;
    a.first[tt.n_blocks] = tiles;
    at = 0;
    for (int q = 0; q <= tt.n_blocks; ++q) {
        const long long end = q < tt.n_blocks ? tt.b[q].off : n;
        if (end > at) {
            a.seg[a.n_seg][0] = at;
            a.seg[a.n_seg][1] = end;
            a.seg0[a.n_seg++] = tiles;
            tiles += (int)((end - at + 2047) / 2048);
        }
        if (q < tt.n_blocks) {
            // a block that does not end on a boundary would share eight parameters with what follows
            if (((long long)tt.b[q].rows * tt.b[q].cols) & 7) return false;
            at = tt.b[q].off + (long long)tt.b[q].rows * tt.b[q].cols;
        }
    }
    a.tiles = tiles;
    *out = a;
    return true;
}

}  // namespace

}  // namespace mcw

using namespace mcw;

extern "C" {

int mcw_mlp_reduce_splits(const float *src, int64_t stride_split, int64_t stride_src, int64_t ld_src, float *dst,
                          int64_t stride_dst, int64_t ld_dst, int32_t splits, int32_t groups, int32_t m, int32_t n,
                          void *stream) {
    if (!src || !dst || splits < 1 || groups < 1 || m < 0 || n < 0) return MCW_MLP_ERR_ARG;
    if (m == 0 || n == 0) return 0;
    const long long total = (long long)m * n;
    const int blocks = (int)((total + 255) / 256 < 1024 ? (total + 255) / 256 : 1024);
    reduce_splits_kernel<<<dim3(blocks, 1, groups), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        src, stride_split, stride_src, ld_src, dst, stride_dst, ld_dst, splits, m, n);
    return cudaGetLastError() == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
}

int mcw_mlp_loss_grouped(const float *y, int64_t ldy, int64_t stride_y, const float *t, int64_t ldt,
                         int64_t stride_t, const float *w, int32_t groups, int32_t m, int32_t n, float *g32,
                         int64_t ldg, int64_t stride_g32, void *g16, int64_t stride_g16, void *g16t, int64_t ldgt,
                         int64_t stride_g16t, float *loss, void *stream) {
    if (!y || !t || !g32 || !g16 || !g16t || !loss || groups < 1 || m < 0 || n < 0) return MCW_MLP_ERR_ARG;
    if (m == 0 || n == 0) return 0;
    const dim3 grid((n + 31) / 32, (m + kLossRows - 1) / kLossRows, groups);
    loss_grouped_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        y, ldy, stride_y, t, ldt, stride_t, w, m, n, g32, ldg, stride_g32, static_cast<__nv_bfloat16 *>(g16),
        stride_g16, static_cast<__nv_bfloat16 *>(g16t), ldgt, stride_g16t, loss);
    return cudaGetLastError() == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
}

int mcw_mlp_colsum_grouped(const McwColsumLayer *layers, int32_t n_layers, int32_t groups, int32_t m, float *out,
                           int64_t stride_out, float *partial, int32_t rows_per_chunk, void *stream) {
    if (!layers || n_layers < 1 || n_layers > 4 || groups < 1 || m < 0 || !out) return MCW_MLP_ERR_ARG;
    ColsumTable tab;
    memset(&tab, 0, sizeof(tab));
    int nmax = 0;
    for (int q = 0; q < n_layers; ++q) {
        if (!layers[q].g || layers[q].n < 0) return MCW_MLP_ERR_ARG;
        tab.l[q].src = layers[q].g;
        tab.l[q].ld = layers[q].ld;
        tab.l[q].s_g = layers[q].stride;
        tab.l[q].off = layers[q].out_offset;
        tab.l[q].n = layers[q].n;
        nmax = layers[q].n > nmax ? layers[q].n : nmax;
    }
    tab.n_layers = n_layers;
    if (nmax == 0) return 0;
    const bool split = partial && rows_per_chunk > 0 && rows_per_chunk < m;
    const int rpc = split ? rows_per_chunk : (m > 0 ? m : 1);
    const int chunks = (m + rpc - 1) / rpc > 0 ? (m + rpc - 1) / rpc : 1;
    if (chunks > 65535 || (long long)n_layers * groups > 65535) return MCW_MLP_ERR_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    colsum_grouped_kernel<<<dim3((nmax + 31) / 32, chunks, n_layers * groups), 256, 0, s>>>(
        tab, groups, m, rpc, out, stride_out, split ? partial : nullptr, nmax);
    if (split)
        colsum_finish_kernel<<<dim3((nmax + 127) / 128, 1, n_layers * groups), 128, 0, s>>>(
            tab, groups, chunks, partial, nmax, out, stride_out);
    return cudaGetLastError() == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
}

int mcw_mlp_adam_grouped(float *w, const float *g, float *m, float *v, void *w16, int64_t n, int32_t groups,
                         const float *lr_dev, const int32_t *step_dev, float beta1, float beta2, float eps,
                         void *wt, int64_t stride_t, const McwTransposeBlock *blocks, int32_t n_blocks,
                         void *stream) {
    if (!w || !g || !m || !v || !w16 || !lr_dev || !step_dev || n < 0 || groups < 1 || n_blocks < 0 ||
        n_blocks > 4 || (n_blocks > 0 && (!blocks || !wt)))
        return MCW_MLP_ERR_ARG;
    if (n == 0) return 0;
    TransposeTable tt;
    memset(&tt, 0, sizeof(tt));
    for (int q = 0; q < n_blocks; ++q) {
        if (blocks[q].offset < 0 || blocks[q].rows < 0 || blocks[q].cols < 0 ||
            blocks[q].offset + (int64_t)blocks[q].rows * blocks[q].cols > n || blocks[q].ld_t < blocks[q].rows)
            return MCW_MLP_ERR_ARG;
        tt.b[q].off = blocks[q].offset;
        tt.b[q].off_t = blocks[q].offset_t;
        tt.b[q].ld_t = blocks[q].ld_t;
        tt.b[q].rows = blocks[q].rows;
        tt.b[q].cols = blocks[q].cols;
    }
    tt.n_blocks = n_blocks;
    AdamTiles at;
    const uintptr_t align = (uintptr_t)w | (uintptr_t)g | (uintptr_t)m | (uintptr_t)v | (uintptr_t)w16 | (uintptr_t)wt;
    if (!(align & 15) && make_adam_tiles(tt, n, stride_t, &at)) {
        const cudaError_t e = launch_after(
            adam_tiled_kernel, dim3((unsigned)at.tiles, groups), 256, 0, static_cast<cudaStream_t>(stream), w, g, m, v,
            static_cast<__nv_bfloat16 *>(w16), n, lr_dev, step_dev, beta1, beta2, eps,
            static_cast<__nv_bfloat16 *>(wt), stride_t, at);
        return e == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
    }
    const dim3 grid((unsigned)((n + 255) / 256), groups);
    adam_grouped_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        w, g, m, v, static_cast<__nv_bfloat16 *>(w16), n, lr_dev, step_dev, beta1, beta2, eps,
        static_cast<__nv_bfloat16 *>(wt), stride_t, tt);
    return cudaGetLastError() == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
}

int mcw_mlp_gather(const void *x_all, const float *t_all, int64_t ldt_all, int32_t n_out, const int32_t *perm,
                   int64_t n_rows, const int32_t *counter_dev, int32_t batch, int32_t groups, void *x,
                   int64_t stride_x, void *xt, int64_t stride_xt, float *t, int64_t ldt, int64_t stride_t,
                   void *stream) {
    if (!x_all || !t_all || !perm || !counter_dev || !x || !xt || !t || batch < 1 || groups < 1 || n_out < 0 ||
        n_rows < batch)
        return MCW_MLP_ERR_ARG;
    gather_kernel<<<dim3(batch, groups), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16 *>(x_all), t_all, ldt_all, n_out, perm, n_rows, counter_dev, batch,
        static_cast<__nv_bfloat16 *>(x), stride_x, static_cast<__nv_bfloat16 *>(xt), stride_xt, t, ldt, stride_t, nullptr);
    return cudaGetLastError() == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
}

int mcw_mlp_step_begin(const void *x_all, const float *t_all, int64_t ldt_all, int32_t n_out, const int32_t *perm,
                       int64_t n_rows, const int32_t *counter_dev, int32_t batch, int32_t groups, void *x,
                       int64_t stride_x, float *t, int64_t ldt, int64_t stride_t, float *loss, void *stream) {
    if (!x_all || !t_all || !perm || !counter_dev || !x || !t || batch < 1 || groups < 1 || n_out < 0 ||
        n_rows < batch)
        return MCW_MLP_ERR_ARG;
    const cudaError_t e = launch_after(
        gather_kernel, dim3(batch, groups), 128, 0, static_cast<cudaStream_t>(stream),
        static_cast<const __nv_bfloat16 *>(x_all), t_all, ldt_all, n_out, perm, n_rows, counter_dev, batch,
        static_cast<__nv_bfloat16 *>(x), stride_x, static_cast<__nv_bfloat16 *>(nullptr), 0, t, ldt, stride_t, loss);
    return e == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
}

int mcw_mlp_advance(int32_t *counter_dev, int32_t *step_dev, void *stream) {
    if (!counter_dev || !step_dev) return MCW_MLP_ERR_ARG;
    const cudaError_t e = launch_after(advance_kernel, 1, 32, 0, static_cast<cudaStream_t>(stream), counter_dev, step_dev);
    return e == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
}

}  // extern "C"
