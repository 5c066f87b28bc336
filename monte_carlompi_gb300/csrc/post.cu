// Post-processing of per-photon records on the device: the reference's BRF and
// albedo arithmetic (post_processing.py:46-100 brf, :102-146 polar BRFs,
// :250-312 spectral albedo; monte_carlo3D.py:1659-1671 calculate_albedo) over
// records already in device memory, instead of re-reading the CSV text.
//
// Per config: the condition-1 exit zenith histogram weighted by wvn with
// np.histogram's binning of [0, pi/2] (edges i * (pi/2)/n, last edge pi/2;
// index ((x - 0) / (pi/2)) * n truncated, then moved one bin down when x is
// below its lower edge and one bin up when x reaches its upper edge, the last bin
// closed), wvn sums per end condition (fixed point 2^-32, so sums do not depend
// on order), counts, and sums of n_scat, path length and wavelength for the
// means the reference prints.
#include <cuda_runtime.h>

#include "mcw_internal.cuh"

namespace mcw {

namespace {

__device__ __forceinline__ int np_bin(double x, int n, double step) {
    const double last = kPi / 2;
    if (!(x >= 0.0) || !(x <= last)) return -1;
    int i = (int)((x / last) * (double)n);
    if (i == n) i -= 1;
    const double lo = (double)i * step;
    const double hi = (i + 1 == n) ? last : (double)(i + 1) * step;
    if (x < lo) i -= 1;
    else if (x >= hi && i != n - 1) i += 1;
    return i;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct PostRec {
    int cond, nscat;
    uint32_t cfg;
    double wvn, path;
    double theta;      // kF64
    float theta32;     // otherwise
    unsigned long long wfx;
};

// vec: FP32 records whose base and stride are multiples of 16 bytes (two 16-byte loads).
template <bool kF64>
__device__ __forceinline__ PostRec load_rec(const char *p, bool vec) {
    PostRec o;
    if (kF64) {
        const mcw_record64 r = *reinterpret_cast<const mcw_record64 *>(p);
        o.cond = r.condition, o.nscat = r.n_scat, o.cfg = r.config;
        o.wvn = r.wvn, o.path = r.path_length, o.theta = r.theta_n, o.theta32 = 0.f;
        o.wfx = (unsigned long long)llrint(r.wvn * 4294967296.0);
    } else {
        float4 u, v;
        if (vec) {
            u = reinterpret_cast<const float4 *>(p)[0], v = reinterpret_cast<const float4 *>(p)[1];
        } else {
            const float *f = reinterpret_cast<const float *>(p);
            u = make_float4(f[0], f[1], f[2], f[3]), v = make_float4(f[4], f[5], f[6], f[7]);
        }
        o.cond = __float_as_int(u.x), o.nscat = __float_as_int(u.y), o.cfg = __float_as_uint(v.w);
        o.wvn = u.z, o.path = v.y, o.theta = 0.0, o.theta32 = u.w;
        o.wfx = (unsigned long long)__float2ll_rn(u.z * 4294967296.f);   // a power of two: exact
    }
    return o;
}

// Totals of one config, straight to global memory (records off the warp's current config).
__device__ __forceinline__ void post_direct(mcw_post_stats *st, const PostRec &r) {
    atomicAdd(reinterpret_cast<unsigned long long *>(&st->q_cond_fx[r.cond]), r.wfx);
    atomicAdd(reinterpret_cast<unsigned long long *>(&st->n_cond[r.cond]), 1ull);
    atomicAdd(reinterpret_cast<unsigned long long *>(&st->sum_n_scat), (unsigned long long)r.nscat);
    atomicAdd(&st->sum_path_length, r.path);
    atomicAdd(&st->sum_wavelength, 1.0 / r.wvn);
}

// A warp's running totals of its current config, a share in every lane's registers.
struct PostSums {
    unsigned long long q[6], nscat;
    unsigned int n[6];
    double path, wvl;
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 1; k < 6; ++k) q[k] = 0, n[k] = 0;
        nscat = 0;
        path = wvl = 0.0;
    }
    __device__ __forceinline__ void add(const PostRec &r) {
#pragma unroll
        for (int k = 1; k < 6; ++k) {
            q[k] += r.cond == k ? r.wfx : 0ull;
            n[k] += r.cond == k ? 1u : 0u;
        }
        nscat += (unsigned long long)r.nscat;
        path += r.path;
        wvl += 1.0 / r.wvn;
    }
    __device__ __forceinline__ void flush(mcw_post_stats *st, int lane) {
        unsigned long long mine = 0;
#pragma unroll
        for (int k = 1; k < 6; ++k) {
            const unsigned long long qs = warp_sum(q[k]);
            const unsigned ns = __reduce_add_sync(0xffffffffu, n[k]);
            if (lane == k) mine = qs;
            if (lane == 8 + k) mine = ns;
        }
        const unsigned long long ss = warp_sum(nscat);
        const double ps = warp_sum(path), ws = warp_sum(wvl);
        if (lane >= 1 && lane < 6 && mine) atomicAdd(reinterpret_cast<unsigned long long *>(&st->q_cond_fx[lane]), mine);
        if (lane >= 9 && lane < 14 && mine)
            atomicAdd(reinterpret_cast<unsigned long long *>(&st->n_cond[lane - 8]), mine);
        if (lane == 6) atomicAdd(reinterpret_cast<unsigned long long *>(&st->sum_n_scat), ss);
        if (lane == 7) atomicAdd(&st->sum_path_length, ps);
        if (lane == 8) atomicAdd(&st->sum_wavelength, ws);
        clear();
    }
};

constexpr int kPostThreads = 256;
constexpr int kPostSmemBins = 2048;   // histograms up to this many bins live in shared memory

// recs: records of stride bytes whose leading fields are an mcw_record64 (kF64) or an
// mcw_record32 (the polarised records extend them).
//
// Bound: one read of the records (32 B each) over the host link, or HBM when they are on the
// device.  Every block takes one contiguous run of records and every warp of it 32 at a time, so
// a record array written config by config keeps a warp on one config: its totals stay in
// registers and go out once per warp and config with warp reductions, the block's zenith
// histogram (of its first record's config) sits in shared memory as 32-bit halves whose carry
// comes from the atomic's old value (the sums stay exact modulo 2^64).  Records of other
// configs, or in no order, take global atomics each.  FP32 zenith angles are binned against
// float thresholds, the smallest float at or above each FP64 edge, which compares as the FP64
// edge does.  A call on one million records of one config in host memory: 4.58 ms with five
// atomics on the config's totals per record, 0.24 ms now (134 GB/s of records, the host link).
template <bool kF64>
__global__ void __launch_bounds__(kPostThreads) post_kernel(const char *recs, size_t stride, int64_t n,
                                                            int64_t per_block, int n_cfg, int n_bins, double step,
                                                            unsigned long long *bins_fx, unsigned int *bins_cnt,
                                                            mcw_post_stats *stats) {
    extern __shared__ unsigned int sh[];     // lo | hi | count | float edges (n_bins + 1)
    const bool hist = n_bins > 0 && n_bins <= kPostSmemBins;
    unsigned int *h_lo = sh, *h_hi = sh + n_bins, *h_cnt = sh + 2 * n_bins;
    float *edge = reinterpret_cast<float *>(sh + 3 * n_bins);
    const int lane = threadIdx.x & 31;
    const int64_t lo = (int64_t)blockIdx.x * per_block;
    const int64_t hi = min(n, lo + per_block);
    if (lo >= hi) return;                    // block-uniform
    const bool vec = ((reinterpret_cast<uintptr_t>(recs) | stride) & 15) == 0;
    if (hist) {
        for (int i = threadIdx.x; i < 3 * n_bins; i += kPostThreads) sh[i] = 0u;
        if (!kF64)
            for (int i = threadIdx.x; i <= n_bins; i += kPostThreads)
                edge[i] = __double2float_ru(i == n_bins ? kPi / 2 : (double)i * step);
        __syncthreads();
    }
    const uint32_t block_cfg = load_rec<kF64>(recs + lo * (int64_t)stride, vec).cfg;
    PostSums sums;
    sums.clear();
    uint32_t cur = 0xffffffffu;              // the warp's config (n_cfg is below 2^31)
    const float guess = (float)((double)n_bins / (kPi / 2));
    for (int64_t base = lo + (threadIdx.x & ~31); base < hi; base += kPostThreads) {
        const int64_t i = base + lane;
        PostRec r;
        r.cond = 0;
        r.cfg = 0;
        if (i < hi) r = load_rec<kF64>(recs + i * (int64_t)stride, vec);
        const bool ok = i < hi && r.cond >= 1 && r.cond <= 5 && r.cfg < (uint32_t)n_cfg;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (!m) continue;
        const uint32_t c0 = __shfl_sync(0xffffffffu, r.cfg, __ffs(m) - 1);
        // the warp moves on to the config of its first record when several records are of it
        if (c0 != cur && __popc(__ballot_sync(0xffffffffu, ok && r.cfg == c0)) >= 8) {
            if (cur != 0xffffffffu) sums.flush(stats + cur, lane);
            cur = c0;
        }
        if (!ok) continue;
        if (r.cfg == cur) sums.add(r);
        else post_direct(stats + r.cfg, r);
        if (r.cond == 1 && n_bins > 0) {
            int b;
            if (!kF64 && hist) {
                const float x = r.theta32;
                b = -1;
                if (x >= 0.f && (double)x <= kPi / 2) {
                    b = min((int)(x * guess), n_bins - 1);
                    while (b > 0 && x < edge[b]) --b;
                    while (b < n_bins - 1 && x >= edge[b + 1]) ++b;
                }
            } else {
                b = np_bin(kF64 ? r.theta : (double)r.theta32, n_bins, step);
            }
            if (b >= 0) {
                if (hist && r.cfg == block_cfg) {
                    const unsigned w_lo = (unsigned)r.wfx, w_hi = (unsigned)(r.wfx >> 32);
                    const unsigned old = atomicAdd(&h_lo[b], w_lo);
                    const unsigned up = w_hi + (old + w_lo < old ? 1u : 0u);
                    if (up) atomicAdd(&h_hi[b], up);
                    atomicAdd(&h_cnt[b], 1u);
                } else {
                    atomicAdd(bins_fx + (size_t)r.cfg * n_bins + b, r.wfx);
                    atomicAdd(bins_cnt + (size_t)r.cfg * n_bins + b, 1u);
                }
            }
        }
    }
    __syncwarp();
    if (cur != 0xffffffffu) sums.flush(stats + cur, lane);
    if (hist) {
        __syncthreads();
        for (int b = threadIdx.x; b < n_bins; b += kPostThreads)
            if (h_cnt[b]) {                  // a non-empty bin's config is below n_cfg
                atomicAdd(bins_fx + (size_t)block_cfg * n_bins + b,
                          ((unsigned long long)h_hi[b] << 32) + h_lo[b]);
                atomicAdd(bins_cnt + (size_t)block_cfg * n_bins + b, h_cnt[b]);
            }
    }
}

}  // namespace

cudaError_t launch_post(const void *recs, bool f64, size_t stride, int64_t n, int n_cfg, int n_bins,
                        unsigned long long *bins_fx, unsigned int *bins_cnt, mcw_post_stats *stats, int sms,
                        cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const double step = (kPi / 2) / (double)(n_bins > 0 ? n_bins : 1);
    // one contiguous run per block, whole rounds of the block, at most four blocks per SM
    const int64_t rounds = (n + kPostThreads - 1) / kPostThreads;
    const int64_t blocks = rounds < (int64_t)sms * 4 ? rounds : (int64_t)sms * 4;
    const int64_t per_block = (rounds + blocks - 1) / blocks * kPostThreads;
    const unsigned grid = (unsigned)((n + per_block - 1) / per_block);
    const size_t smem = n_bins > 0 && n_bins <= kPostSmemBins ? (size_t)(4 * n_bins + 1) * 4 : 0;
    const char *p = static_cast<const char *>(recs);
    if (f64)
        post_kernel<true><<<grid, kPostThreads, smem, s>>>(p, stride, n, per_block, n_cfg, n_bins, step, bins_fx,
                                                           bins_cnt, stats);
    else
        post_kernel<false><<<grid, kPostThreads, smem, s>>>(p, stride, n, per_block, n_cfg, n_bins, step, bins_fx,
                                                            bins_cnt, stats);
    return cudaGetLastError();
}

}  // namespace mcw
