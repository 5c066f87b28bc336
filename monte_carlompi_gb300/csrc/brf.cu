// From the surrogate's standardised outputs to BRFs, in FP64: members' BRFs, their mean and
// spread, a retrieval's costs and Gauss-Newton sums.  Compiled with --fmad=false: every product
// and sum is rounded on its own, in the order of the array code these kernels took the place of
// (surrogate.from_target, Ensemble.predict, inverse.surrogate_gn), but where one is written as fma, means
// over the members divided.
//
// Target space: y * std + mean = log(BRF / albedo + floor) for the 648 bins and log(albedo).
//
// What bounds them: FP64 (64 cycles a warp an operation on a sub-core), so every kernel takes each
// exponential once, eleven operations by table, divides once where it can, and keeps what it can in
// registers; a block per row, a thread per bin, sums by block reduction.  16 grid points of 128
// observations, five members: 362 us with CUDA's exp and a division a weight a point, 285 now; a
// Jacobian 46 now (259 and 44 with exponentials of 1.24 ulp, the floors taken off a sum and means by the
// reciprocal, which lost digits).  One retrieval of 128 observations with five members (16-point grid, six
// iterations, spreads): 92 ms on the host's cores and elementwise tensor kernels; 3.3 ms with these kernels and the steps and the encoding of log r on the host, a
// wait for the device and two copies an iteration; 1.55 ms with the steps here too and the network
// laid out while the grid's costs are worked out.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/mcw_mlp.h"
#include "smem_limit.cuh"

namespace mcw {

namespace {

constexpr int kBins = MCW_MLP_OUT - 1;     // 648
constexpr int kThreads = 224;              // 7 warps, three bins a thread (672)
constexpr int kPer = 3;

// Block sum (every thread gets it); `red` holds one value per warp.
__device__ __forceinline__ double block_sum(double v, double *red) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = red[0];
#pragma unroll
    for (int q = 1; q < kThreads / 32; ++q) s += red[q];
    return s;
}

// exp(x) by table (Tang, ACM Trans. Math. Softw. 15, 1989): x = (64 k + j) ln 2 / 64 + r, |r| <= a = ln 2 /
// 128, so exp(x) = 2^k 2^(j / 64) exp(r), the power as the sum of two doubles.  Of exp(r)'s series five
// terms, the sixth, r^6 / 720, put into those of r^4 and r^2 (its Chebyshev expansion on [-a, a]: x^6 = 3/2
// a^2 x^4 - 9/16 a^4 x^2 but for a^6 / 16), which leaves 3e-18.  Eleven FP64 operations, all these kernels
// are bound by; past +-700 CUDA's exp.  Within 0.55 ulp of the exact value; CUDA's exp 0.88, and with
// 2^(j / 64) as one double and the plain series, ten operations, 1.24 (a retrieval of 128 observations
// 1.54 ms, 1.55 now).
__device__ const double2 kExp2[64] = {
    {0x1.0000000000000p+0, 0}, {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55}, {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54}, {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54}, {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55}, {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54}, {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55}, {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59}, {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55}, {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54}, {0x1.6623882552225p+0, -0x1.bb60987591c34p-54},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}, {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55}, {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54}, {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57}, {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56}, {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54}, {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56}, {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56}, {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55}, {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54}, {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54}, {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55},
};
__device__ __forceinline__ double exp_by_table(double x, const double2 *tab) {
    if ((__double2hiint(x) & 0x7fffffff) >= 0x4085e000) return exp(x);
    const double t = fma(x, 0x1.71547652b82fep+6, 0x1.8p52);
    const int n = __double2loint(t);
    const double m = t - 0x1.8p52;
    const double r = fma(-m, 0x1.abc9e3b39803fp-62, fma(-m, 0x1.62e42fefa39efp-7, x));
    double q = fma(r, 1.0 / 120.0, 0x1.55557621dbbb3p-5);    // 1 / 24 + 3/2 a^2 / 720
    q = fma(q, r, 1.0 / 6.0);
    q = fma(q, r, 0x1.fffffffffd0bap-2);                     // 1 / 2 - 9/16 a^4 / 720
    const double2 T = tab[n & 63];
    const double y = T.x + fma(T.x, fma(q, r * r, r), T.y);
    return __hiloint2double(__double2hiint(y) + ((n >> 6) << 20), __double2loint(y));
}
// The table in shared memory (the caller's barrier follows); a row's one albedo takes it from kExp2.
__device__ __forceinline__ void load_exp2(double2 *tab) {
    if (threadIdx.x < 64) tab[threadIdx.x] = kExp2[threadIdx.x];
}

__device__ __forceinline__ double unscaled(double y, double std, double mean) { return y * std + mean; }

// BRF of one bin: (exp(y) - floor) * albedo.
__device__ __forceinline__ double bin_brf(const __half *row, int b, const double *std, const double *mean, double floor,
                                          double albedo, const double2 *tab) {
    return (exp_by_table(unscaled((double)__half2float(row[b]), std[b], mean[b]), tab) - floor) * albedo;
}

__device__ __forceinline__ double row_albedo(const __half *row, const double *std, const double *mean) {
    return exp_by_table(unscaled((double)__half2float(row[kBins]), std[kBins], mean[kBins]), kExp2);
}

// t / members, correctly rounded, share = 1 / members: the residual's correction (Markstein, IBM J. Res.
// Dev. 34, 1990).  With a whole number of at most 14 bits below the line the residual is exact, and the
// quotient at least ulp / (2 members) from the middle between two doubles, or a double.
__device__ __forceinline__ double mean_of(double t, int members, double share) {
    const double q = t * share, s = fma(fma(-q, (double)members, t), share, q);
    return (__double2hiint(q) & 0x7fffffff) < 0x7ff00000 ? s : q;
}

// The larger of x and lo; NaN stays NaN.
__device__ __forceinline__ double at_least(double x, double lo) { return x < lo ? lo : x; }

// Weight of a bin's residual: 1 / variance (counting noise of `photons`, relative noise, the
// model's variance), or the bin's share without photons.
struct Noise {
    double photons, rel;
    const double *share;       // [648]
    const double *rel_bins;    // relative noise per row and bin [n, 648] in place of rel, or null
    __device__ __forceinline__ double variance(double f, double model, int r, int b) const {
        const double q = rel_bins ? rel_bins[(size_t)r * kBins + b] : rel;
        const double v = at_least(f, 1e-3) / (photons * share[b]) + (q * f) * (q * f);
        return v + model;
    }
};

// Each member's BRF and albedo of row blockIdx.x.
__global__ void __launch_bounds__(kThreads) members_kernel(const __half *ys, long long pitch, int n, const double *mean,
                                                           const double *std, double floor, double *brf, double *alb) {
    const int r = blockIdx.x, m = blockIdx.y;
    const __half *row = ys + ((size_t)m * n + r) * pitch;
    const double *mu = mean + (size_t)m * (kBins + 1), *sd = std + (size_t)m * (kBins + 1);
    __shared__ double a;
    __shared__ double2 tab[64];
    load_exp2(tab);
    if (threadIdx.x == 0) {
        a = row_albedo(row, sd, mu);
        alb[(size_t)m * n + r] = a;
    }
    __syncthreads();
    for (int b = threadIdx.x; b < kBins; b += kThreads)
        brf[((size_t)m * n + r) * kBins + b] = bin_brf(row, b, sd, mu, floor, a, tab);
}

// Mean BRF and albedo over the members, and the spread: the weighted RMS of the members' standard
// deviation over the weighted RMS of the mean.
__global__ void __launch_bounds__(kThreads) stats_kernel(const double *brf, const double *alb, int members, int n,
                                                         const double *share, double *mean, double *alb_mean,
                                                         double *spread) {
    __shared__ double red[kThreads / 32];
    const int r = blockIdx.x;
    double num = 0.0, den = 0.0;
    for (int b = threadIdx.x; b < kBins; b += kThreads) {
        const double *p = brf + (size_t)r * kBins + b;
        const size_t s = (size_t)n * kBins;
        double t = 0.0;
        for (int m = 0; m < members; ++m) t += p[m * s];
        const double mu = t / members;
        double v = 0.0;
        for (int m = 0; m < members; ++m) {
            const double d = p[m * s] - mu;
            v += d * d;
        }
        mean[(size_t)r * kBins + b] = mu;
        num += v / members * share[b];
        den += mu * mu * share[b];
    }
    num = block_sum(num, red);
    den = block_sum(den, red);
    if (threadIdx.x == 0) {
        spread[r] = sqrt(num / at_least(den, 1e-30));
        double t = 0.0;
        for (int m = 0; m < members; ++m) t += alb[(size_t)m * n + r];
        alb_mean[r] = t / members;
    }
}

// Cost of a grid point for an observation: sum over bins of w (mean BRF - obs)^2, w from the
// observation's own noise, taken once for the block's points.  Row point * n_obs + observation.
__global__ void __launch_bounds__(kThreads) cost_kernel(const __half *ys, long long pitch, int members, int points, int per,
                                                        int n_obs, const double *mean, const double *std, double floor,
                                                        const double *obs, const Noise noise, double *cost) {
    extern __shared__ double albs[];         // members, of the block's points
    __shared__ double red[kThreads / 32];
    __shared__ double2 tab[64];
    const int o = blockIdx.x % n_obs, p0 = blockIdx.x / n_obs * per, np = min(per, points - p0), rows = points * n_obs;
    load_exp2(tab);
    for (int q = threadIdx.x; q < members * np; q += kThreads) {
        const int m = q % members, r = (p0 + q / members) * n_obs + o;
        albs[q] = row_albedo(ys + ((size_t)m * rows + r) * pitch, std + (size_t)m * (kBins + 1), mean + (size_t)m * (kBins + 1));
    }
    __syncthreads();
    const double share = 1.0 / members;
    double x[kPer], w[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int b = threadIdx.x + k * kThreads;
        x[k] = w[k] = 0.0;
        if (b < kBins) {
            x[k] = obs[(size_t)o * kBins + b];
            w[k] = noise.photons != 0 ? 1.0 / noise.variance(x[k], 0.0, o, b) : noise.share[b];
        }
    }
    for (int p = 0; p < np; ++p) {
        const int r = (p0 + p) * n_obs + o;
        double c = 0.0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int b = threadIdx.x + k * kThreads;
            if (b >= kBins) break;
            double t = 0.0;
            for (int m = 0; m < members; ++m) {
                const double *mu = mean + (size_t)m * (kBins + 1), *sd = std + (size_t)m * (kBins + 1);
                const double y = (double)__half2float(ys[((size_t)m * rows + r) * pitch + b]);
                t = fma(exp_by_table(fma(y, sd[b], mu[b]), tab) - floor, albs[p * members + m], t);
            }
            const double d = mean_of(t, members, share) - x[k];
            c += w[k] * (d * d);
        }
        c = block_sum(c, red);
        if (threadIdx.x == 0) cost[r] = c;
    }
}

// Mean BRF f, d f / d log r (j) and the members' variance (v) of row blockIdx.x from the outputs y
// and their tangents, FP32 [members, n, pitch]; any of f_out, j_out, v_out may be null.  With obs:
// the Gauss-Newton sums over the bins of w j (f - obs) and w j^2.
__global__ void __launch_bounds__(kThreads) jacobian_kernel(const float *y, const float *ydot, long long pitch, int members,
                                                            int n, const double *mean, const double *std, double floor,
                                                            double *f_out, double *j_out, double *v_out,
                                                            const double *obs, const Noise noise, double *jtr, double *jtj) {
    extern __shared__ double sh[];           // albedo and its slope per member
    __shared__ double red[kThreads / 32];
    __shared__ double2 tab[64];
    const int r = blockIdx.x;
    const double each = 1.0 / members;
    load_exp2(tab);
    for (int m = threadIdx.x; m < members; m += kThreads) {
        const size_t at = ((size_t)m * n + r) * pitch + kBins;
        const double sd = std[(size_t)m * (kBins + 1) + kBins];
        const double a = exp_by_table(unscaled((double)y[at], sd, mean[(size_t)m * (kBins + 1) + kBins]), kExp2);
        sh[2 * m] = a;
        sh[2 * m + 1] = a * ((double)ydot[at] * sd);
    }
    __syncthreads();
    double sr = 0.0, sj = 0.0;
    for (int b = threadIdx.x; b < kBins; b += kThreads) {
        double f = 0.0, j = 0.0, f2 = 0.0;
        for (int m = 0; m < members; ++m) {
            const size_t at = ((size_t)m * n + r) * pitch + b;
            const double sd = std[(size_t)m * (kBins + 1) + b], a = sh[2 * m];
            const double shape = exp_by_table(fma((double)y[at], sd, mean[(size_t)m * (kBins + 1) + b]), tab);
            const double dp = (double)ydot[at] * sd;
            const double fm = (shape - floor) * a;
            f += fm;
            f2 += fm * fm;
            j += shape * dp * a + (shape - floor) * sh[2 * m + 1];
        }
        f = mean_of(f, members, each);
        j = mean_of(j, members, each);
        const double v = at_least(mean_of(f2, members, each) - f * f, 0.0);
        if (f_out) f_out[(size_t)r * kBins + b] = f;
        if (j_out) j_out[(size_t)r * kBins + b] = j;
        if (v_out) v_out[(size_t)r * kBins + b] = v;
        if (obs) {
            const double d = f - obs[(size_t)r * kBins + b];
            const double w = noise.photons != 0 ? 1.0 / noise.variance(f, v, r, b) : noise.share[b];
            sr += w * j * d;
            sj += w * j * j;
        }
    }
    if (!obs) return;
    sr = block_sum(sr, red);
    sj = block_sum(sj, red);
    if (threadIdx.x == 0) {
        jtr[r] = sr;
        jtj[r] = sj;
    }
}

// The members' standard deviation of log r at the solution (inverse.logr_spread) and the posterior
// width the observation noise alone allows, 1 / sqrt(sum j^2 / var).
__global__ void __launch_bounds__(kThreads) logr_kernel(const double *brf, const double *mean, int members, int n,
                                                        const double *f, const double *j, const double *v,
                                                        const Noise noise, double *spread, double *sigma) {
    __shared__ double red[kThreads / 32];
    const int r = blockIdx.x;
    double wj[kPer], mu[kPer];
    double sj = 0.0, sn = 0.0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int b = threadIdx.x + k * kThreads;
        wj[k] = mu[k] = 0.0;
        if (b < kBins) {
            const size_t at = (size_t)r * kBins + b;
            const double w = noise.photons != 0 ? 1.0 / noise.variance(f[at], v[at], r, b) : noise.share[b];
            const double wn = noise.photons != 0 ? 1.0 / noise.variance(f[at], 0.0, r, b) : noise.share[b];
            mu[k] = mean[at];
            wj[k] = w * j[at];
            sj += wj[k] * j[at];
            sn += wn * j[at] * j[at];
        }
    }
    sj = at_least(block_sum(sj, red), 1e-300);
    sn = at_least(block_sum(sn, red), 1e-300);
    // two passes over the members' shifts: their mean, then their deviation
    double total = 0.0, var = 0.0;
    for (int pass = 0; pass < 2; ++pass)
        for (int m = 0; m < members; ++m) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                const int b = threadIdx.x + k * kThreads;
                if (b < kBins) s += wj[k] * (brf[((size_t)m * n + r) * kBins + b] - mu[k]);
            }
            const double ds = block_sum(s, red) / sj;
            if (pass == 0) {
                total += ds;
            } else {
                const double d = ds - total / members;
                var += d * d;
            }
        }
    if (threadIdx.x == 0) {
        spread[r] = sqrt(var / members);
        sigma[r] = 1.0 / sqrt(sn);
    }
}

// The network's inputs, scaled to [-1, 1] over the training hull (surrogate.encode): log r_eff,
// wavelength, mu0, log depth, each (x - origin) over the width.
struct Hull {
    double origin[4], width[4];
    __device__ __forceinline__ float scaled(int q, double x) const { return (float)(2 * (x - origin[q]) / width[q] - 1); }
    __device__ __forceinline__ float4 encode(double s, const double *known) const {
        return make_float4(scaled(0, log(exp(s))), scaled(1, known[0]), scaled(2, known[1]), scaled(3, log(known[2])));
    }
};

// Row p * n + o: observation o at log r = s[p].
__global__ void encode_kernel(const double *s, int points, int n, const double *known, const Hull hull, float4 *x) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row < points * n) x[row] = hull.encode(s[row / n], known + 3 * (row % n));
}

__device__ __forceinline__ double clipped(double x, double lo, double hi) { return x < lo ? lo : (x > hi ? hi : x); }

// log r of every observation: the grid point of the lowest cost, or a damped Gauss-Newton step from
// where it is; then the network's inputs there, FP32 (x) and bf16 for every member (x16, rows of 8),
// either may be null.
__global__ void gn_kernel(const double *cost, const double *grid, int points, const double *jtr, const double *jtj,
                          double damping, double max_step, double lo, double hi, const double *known, int n,
                          const Hull hull, double *s, float4 *x, __nv_bfloat16 *x16, int members) {
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= n) return;
    double at;
    if (cost) {
        double best = __longlong_as_double(0x7ff0000000000000ll);
        at = 0.0;
        for (int p = 0; p < points; ++p) {
            const double c = cost[(size_t)p * n + o];
            if (c < best) best = c, at = grid[p];
        }
    } else {
        const double step = clipped(-jtr[o] / (jtj[o] * (1 + damping) + 1e-30), -max_step, max_step);
        at = clipped(s[o] + step, lo, hi);
    }
    s[o] = at;
    const float4 e = hull.encode(at, known + 3 * (size_t)o);
    if (x) x[o] = e;
    if (x16)
        for (int m = 0; m < members; ++m) {
            __nv_bfloat162 *d = reinterpret_cast<__nv_bfloat162 *>(x16 + ((size_t)m * n + o) * 8);
            d[0] = __floats2bfloat162_rn(e.x, e.y);
            d[1] = __floats2bfloat162_rn(e.z, e.w);
        }
}

Hull hull_of(const double *h) {
    Hull r;
    for (int q = 0; q < 4; ++q) r.origin[q] = h[2 * q], r.width[q] = h[2 * q + 1];
    return r;
}

// The Jacobian keeps 16 bytes a member in shared memory, the costs 8: 200 KB of the 227 at the most.
constexpr int kMaxMembers = 12800;
bool rows_ok(int32_t members, int32_t n) { return members >= 1 && members <= kMaxMembers && n >= 0; }
int done() { return cudaGetLastError() == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA; }

int cost(const void *ys, int64_t pitch, int32_t members, int32_t points, int32_t n_obs, const double *mean,
         const double *std, double floor, const double *obs, const Noise &noise, double *cost, void *stream) {
    if (!ys || !mean || !std || !obs || !noise.share || !cost || points < 0 || n_obs < 0 ||
        (long long)points * n_obs > 0x7fffffffLL || !rows_ok(members, points * n_obs) || pitch < MCW_MLP_OUT)
        return MCW_MLP_ERR_ARG;
    if (points * n_obs == 0) return 0;
    const int per = members <= 1024 ? 4 : 1;       // points a block, within 32 KB of albedos for the usual ensembles
    const size_t smem = per * members * sizeof(double);
    if (smem > 40 * 1024 && allow_smem(reinterpret_cast<const void *>(cost_kernel), kMaxMembers * sizeof(double)) != cudaSuccess)
        return MCW_MLP_ERR_CUDA;
    cost_kernel<<<(points + per - 1) / per * n_obs, kThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half *>(ys), pitch, members, points, per, n_obs, mean, std, floor, obs, noise, cost);
    return done();
}

int jacobian(const float *y, const float *ydot, int64_t pitch, int32_t members, int32_t n, const double *mean,
             const double *std, double floor, double *f, double *j, double *v, const double *obs, const Noise &noise,
             double *jtr, double *jtj, void *stream) {
    if (!y || !ydot || !mean || !std || !rows_ok(members, n) || pitch < MCW_MLP_OUT ||
        (obs && (!noise.share || !jtr || !jtj)))
        return MCW_MLP_ERR_ARG;
    if (n == 0) return 0;
    const size_t smem = 2 * members * sizeof(double);
    if (smem > 40 * 1024 && allow_smem(reinterpret_cast<const void *>(jacobian_kernel), kMaxMembers * 2 * sizeof(double)) != cudaSuccess)
        return MCW_MLP_ERR_CUDA;
    jacobian_kernel<<<n, kThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        y, ydot, pitch, members, n, mean, std, floor, f, j, v, obs, noise, jtr, jtj);
    return done();
}

int logr(const double *brf, const double *mean_brf, int32_t members, int32_t n, const double *f, const double *j,
         const double *v, const Noise &noise, double *spread, double *sigma, void *stream) {
    if (!brf || !mean_brf || !f || !j || !v || !noise.share || !spread || !sigma || !rows_ok(members, n))
        return MCW_MLP_ERR_ARG;
    if (n == 0) return 0;
    logr_kernel<<<n, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(brf, mean_brf, members, n, f, j, v, noise,
                                                                       spread, sigma);
    return done();
}

}  // namespace

}  // namespace mcw

using namespace mcw;

extern "C" {

int mcw_brf_members(const void *ys, int64_t pitch, int32_t members, int32_t n, const double *mean, const double *std,
                    double floor, double *brf, double *albedo, void *stream) {
    if (!ys || !mean || !std || !brf || !albedo || !rows_ok(members, n) || pitch < MCW_MLP_OUT) return MCW_MLP_ERR_ARG;
    if (n == 0) return 0;
    members_kernel<<<dim3(n, members), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half *>(ys), pitch, n, mean, std, floor, brf, albedo);
    return done();
}

int mcw_brf_stats(const double *brf, const double *albedo, int32_t members, int32_t n, const double *share,
                  double *mean_brf, double *mean_albedo, double *spread, void *stream) {
    if (!brf || !albedo || !share || !mean_brf || !mean_albedo || !spread || !rows_ok(members, n)) return MCW_MLP_ERR_ARG;
    if (n == 0) return 0;
    stats_kernel<<<n, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(brf, albedo, members, n, share, mean_brf,
                                                                        mean_albedo, spread);
    return done();
}

int mcw_brf_cost(const void *ys, int64_t pitch, int32_t members, int32_t points, int32_t n_obs, const double *mean,
                 const double *std, double floor, const double *obs, const double *share, double photons,
                 double rel_noise, double *out, void *stream) {
    return cost(ys, pitch, members, points, n_obs, mean, std, floor, obs, Noise{photons, rel_noise, share, nullptr}, out,
                stream);
}

int mcw_brf_cost_noise(const void *ys, int64_t pitch, int32_t members, int32_t points, int32_t n_obs,
                       const double *mean, const double *std, double floor, const double *obs, const double *share,
                       double photons, const double *rel_noise, double *out, void *stream) {
    if (!rel_noise) return MCW_MLP_ERR_ARG;
    return cost(ys, pitch, members, points, n_obs, mean, std, floor, obs, Noise{photons, 0.0, share, rel_noise}, out,
                stream);
}

int mcw_brf_jacobian(const float *y, const float *ydot, int64_t pitch, int32_t members, int32_t n, const double *mean,
                     const double *std, double floor, double *f, double *j, double *v, const double *obs,
                     const double *share, double photons, double rel_noise, double *jtr, double *jtj, void *stream) {
    return jacobian(y, ydot, pitch, members, n, mean, std, floor, f, j, v, obs,
                    Noise{photons, rel_noise, share, nullptr}, jtr, jtj, stream);
}

int mcw_brf_jacobian_noise(const float *y, const float *ydot, int64_t pitch, int32_t members, int32_t n,
                           const double *mean, const double *std, double floor, double *f, double *j, double *v,
                           const double *obs, const double *share, double photons, const double *rel_noise, double *jtr,
                           double *jtj, void *stream) {
    if (!rel_noise) return MCW_MLP_ERR_ARG;
    return jacobian(y, ydot, pitch, members, n, mean, std, floor, f, j, v, obs, Noise{photons, 0.0, share, rel_noise},
                    jtr, jtj, stream);
}

int mcw_brf_encode(const double *s, int32_t points, const double *known, int32_t n, const double *hull, float *x,
                   void *stream) {
    if (!s || !known || !hull || !x || points < 0 || n < 0 || (long long)points * n > 0x7fffffffLL - 128 ||
        (reinterpret_cast<uintptr_t>(x) & 15))
        return MCW_MLP_ERR_ARG;
    if (points * n == 0) return 0;
    encode_kernel<<<(points * n + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(
        s, points, n, known, hull_of(hull), reinterpret_cast<float4 *>(x));
    return done();
}

int mcw_brf_gn_step(const double *cost, const double *grid, int32_t points, const double *jtr, const double *jtj,
                    double damping, double max_step, double lo, double hi, const double *known, int32_t n,
                    const double *hull, double *s, float *x, void *x16, int32_t members, void *stream) {
    if (!known || !hull || !s || n < 0 || n > 0x7fffffff - 128 || members < 0 || (cost ? !grid || points < 0 : !jtr || !jtj) ||
        (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(x16) & 15))
        return MCW_MLP_ERR_ARG;
    if (n == 0) return 0;
    gn_kernel<<<(n + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(
        cost, grid, points, jtr, jtj, damping, max_step, lo, hi, known, n, hull_of(hull), s,
        reinterpret_cast<float4 *>(x), static_cast<__nv_bfloat16 *>(x16), members);
    return done();
}

int mcw_brf_logr(const double *brf, const double *mean_brf, int32_t members, int32_t n, const double *f, const double *j,
                 const double *v, const double *share, double photons, double rel_noise, double *spread, double *sigma,
                 void *stream) {
    return logr(brf, mean_brf, members, n, f, j, v, Noise{photons, rel_noise, share, nullptr}, spread, sigma, stream);
}

int mcw_brf_logr_noise(const double *brf, const double *mean_brf, int32_t members, int32_t n, const double *f,
                       const double *j, const double *v, const double *share, double photons, const double *rel_noise,
                       double *spread, double *sigma, void *stream) {
    if (!rel_noise) return MCW_MLP_ERR_ARG;
    return logr(brf, mean_brf, members, n, f, j, v, Noise{photons, 0.0, share, rel_noise}, spread, sigma, stream);
}

}  // extern "C"
