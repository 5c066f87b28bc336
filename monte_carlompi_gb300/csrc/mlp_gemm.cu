// The surrogate network's GEMM on the 5th-generation tensor cores, every operand tile
// fetched by TMA: C = A B^T for up to four problems in one launch, each for `groups`
// independent products (ensemble members), bf16 operands stored with either dimension
// contiguous, FP32 accumulation in tensor memory.
//
// One CTA of six warps computes a 128 x TN tile.  Warp 4 copies K chunks of 64 through a
// shared-memory ring (cp.async.bulk.tensor.3d, mbarrier transaction counts), warp 5 owns the
// tensor memory and issues tcgen05.mma (128 x TN x 16, K ascending), handing each stage back by
// tcgen05.commit; warps 0-3 run the epilogue, whose other inputs (pre-activations, targets) are
// already in flight while the product runs.
//
// What bounds it: at the network's sizes (K of 256 to 649, or a long K with few tiles) a
// CTA's life is the copies' latency and rate.  So
//  * every box row is 128 bytes (64 bf16 in the 128-byte swizzle; 64 bytes for a transposed
//    operand 32 wide): the 16-byte-wide boxes used before, one per core-matrix column, took a
//    TMA request per 16 bytes and 42 us for a 256 x 256 x 649 product of five members;
//  * an operand stored transposed ([k, m]) is read as MN-major by the tensor core itself, so
//    nothing is transposed on the way (staging it by threads, two bytes at a time, took 7.2 ms
//    for the weight gradient of 65,536 rows);
//  * the copying and the issuing loops are run by whole warps, one elected lane issuing: under
//    `lane == 0` every tcgen05.mma took about 200 cycles to issue (its descriptors had to be moved
//    into uniform registers; a chain of 1,024 chunks 440 us, then 201), and the next stage's
//    barrier is looked at before a stage's MMAs are issued;
//  * tiles are 64 or 32 columns wide, so that four CTAs share an SM or a small product is spread
//    over more SMs (the rules in launch_batch have the times).
// The epilogue goes through a 32 x 32 tile per warp once: a lane then holds one output column of
// 32 rows, so loads and stores are whole row runs, and bias gradients are the lane's running sum.
// At large sizes it is what bounds the launch, by its instructions: a block with all its rows and
// columns has an instance without predicates, its pointers moving a row at a time; with 16-bit
// outputs and even strides a lane takes two columns of every other row; and the SiLU' quotient
// takes five instructions instead of a division.  Instructions an element 47 -> 28 with a bias and
// SiLU, 96 -> 50 with SiLU', 26 -> 18 for the output; the autograd pass of 65,536 rows 742 -> 591 us
// with the stages below, the ensemble's training step 92 -> 76 us.
//
// Every mbarrier wait is bounded (2 s of %globaltimer); a wait that runs out raises bit 2 of
// mcw_mlp_status, the CTA waits (bounded) for its copies and MMAs in flight, frees its tensor
// memory and leaves.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>

#include "../../include/mcw_mlp.h"
#include "pdl.cuh"
#include "rounded.cuh"
#include "smem_limit.cuh"

namespace mcw {

unsigned int *tc_err_flag();

namespace {

constexpr int TM = 128, TK = 64;
constexpr int kMaxStages = 8;
constexpr int kABytes = TM * TK * 2;              // 16 KB
constexpr int kPitch = 34;                        // floats a row of an epilogue warp's 32 x 32 tile
constexpr int kTileBytes = 32 * kPitch * 4;
constexpr int kThreads = 192;
constexpr unsigned long long kWaitNs = 2000000000ull;

__host__ __device__ constexpr int stage_bytes(int tn) { return kABytes + tn * TK * 2; }

// One problem of a launch; CTAs [cta0, cta0 + tiles) are its, and from sum0 those of its column sums.
struct GemmProb {
    CUtensorMap ta, tb;
    int32_t m, n, k, nt, mt;
    int32_t splits, kps, cta0, sum0; // K per split (a multiple of TK)
    const float *bias;
    long long s_bias;
    const float *aux;               // DSILU: pre-activations; LOSS: targets
    long long ld_aux, s_aux;
    void *c;
    long long ldc, s_c, s_split;
    float *c2;
    long long ldc2, s_c2;
    __nv_bfloat16 *ct;
    long long ldct, s_ct;
    float *colsum;                  // SILU'/LOSS: column sums of every 128 rows; F32: their total, out
    const float *colsum_in;         // F32: the column sums of the A operand's rows, or the f32 rows themselves
    long long s_colsum, ld_colsum;  // per group; per 128 rows (per row)
    int32_t colsum_chunks, colsum_rows;
    const float *weights;           // LOSS: per column
    float *loss;                    // LOSS: per group
    int32_t pairs;                  // 16-bit outputs, and what goes with them, on pairs of columns
};

struct GemmBatch {
    GemmProb p[MCW_GEMM_BATCH_MAX];
    unsigned int *err;
    int32_t np, stages, sub, sums0; // K chunks a stage; the first CTA of column sums
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ float silu(float z) { return __fdividef(z, 1.f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
    const float s = reciprocal_rn(1.f + __expf(-z));
    return s * (1.f + z * (1.f - s));
}

__device__ __forceinline__ bool try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}

// Whether the phase has completed, without waiting.
__device__ __forceinline__ bool test_wait(uint64_t *bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}

// Bounded wait; gives up when another role of the CTA has given up, and raises the CTA's abort
// flag when its own time runs out.
__device__ __forceinline__ bool wait_bar(uint64_t *bar, uint32_t parity, volatile int *abort) {
    unsigned long long t0 = 0;
    for (unsigned tries = 1; !try_wait(bar, parity); ++tries) {
        if (tries & 63u) continue;
        if (*abort) return false;
        const unsigned long long t = now_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > kWaitNs) {
            *abort = 1;
            return false;
        }
    }
    return true;
}

// The same by a whole warp, with one verdict.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort) {
    return __all_sync(0xffffffffu, wait_bar(bar, parity, abort));
}

// Bounded wait that ignores the abort flag (draining copies and MMAs in flight).
__device__ __forceinline__ void drain_bar(uint64_t *bar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (unsigned tries = 1; !try_wait(bar, parity); ++tries) {
        if (tries & 63u) continue;
        const unsigned long long t = now_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > kWaitNs) return;
    }
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z,
                                            uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
        :: "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// One lane of the converged warp, the same each time (its MMAs and commits are one sequence).
// The loops around it are run by the whole warp, so descriptors and addresses stay in uniform
// registers.
__device__ __forceinline__ bool elect_one() {
    uint32_t yes;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(yes));
    return yes != 0;
}

__device__ __forceinline__ void commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                 :: "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void bar_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(bar)));
}

// Shared-memory matrix descriptor: start >> 4 (bits 0-13), leading byte offset >> 4 (bits 16-29),
// stride byte offset >> 4 (bits 32-45), version 1 (bit 46), swizzle (bits 61-63: 2 = 128 bytes,
// 4 = 64 bytes).
//  K-major, 128-byte rows of 64 k: eight rows are an atom of 1,024 bytes (stride offset); a
//  K step of 16 is 32 bytes further in the row.
//  MN-major, rows of 64 (32) m or n per k: eight k are an atom of 1,024 (512) bytes (stride
//  offset), the next 64 m or n lie one 64-k box (8,192 bytes) further (leading offset); a K step
//  of 16 is two atoms.
__device__ __forceinline__ uint64_t desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t swizzle) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46) | ((uint64_t)swizzle << 61);
}

template <bool kMn, int kRows>
__device__ __forceinline__ uint64_t operand_desc(uint32_t base, int step) {
    if (!kMn) return desc(base + 32u * step, 16, 1024, 2);
    return kRows >= 64 ? desc(base + 2048u * step, 8192, 1024, 2) : desc(base + 1024u * step, 16, 512, 4);
}

// The copies of a 64-k chunk of kRows rows of one operand.
template <bool kMn, int kRows>
__device__ __forceinline__ void load_operand(uint32_t dst, const CUtensorMap *map, int k0, int row0, int g,
                                             uint64_t *bar) {
    if (!kMn) {
        tma_load_3d(dst, map, k0, row0, g, bar);
    } else {
#pragma unroll
        for (int j = 0; j < (kRows + 63) / 64; ++j) tma_load_3d(dst + j * 8192, map, row0 + 64 * j, k0, g, bar);
    }
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
          "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
          "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
          "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr) : "memory");
}

// The other input of a 32 x 32 block, one column per lane: rows rbase .. rbase + 31 of column
// `col` (pre-activations or targets); all loads in flight at once.
__device__ __forceinline__ void load_aux(const GemmProb &p, int g, int rbase, int col, bool full, float (&av)[32]) {
    const float *src = p.aux + (size_t)g * p.s_aux + (size_t)rbase * p.ld_aux + col;
    if (full) {
#pragma unroll
        for (int r = 0; r < 32; ++r, src += p.ld_aux) av[r] = __ldg(src);
    } else {
#pragma unroll
        for (int r = 0; r < 32; ++r, src += p.ld_aux) av[r] = (col < p.n && rbase + r < p.m) ? __ldg(src) : 0.f;
    }
}

// The same for block_pairs: rows 2 i + lane / 16, two columns a lane.
__device__ __forceinline__ void load_aux_pairs(const GemmProb &p, int g, int rbase, int nb, int lane, float (&av)[32]) {
    const float *src = p.aux + (size_t)g * p.s_aux + (size_t)(rbase + (lane >> 4)) * p.ld_aux + nb + 2 * (lane & 15);
#pragma unroll
    for (int i = 0; i < 16; ++i, src += 2 * p.ld_aux) {
        const float2 v = __ldg(reinterpret_cast<const float2 *>(src));
        av[2 * i] = v.x, av[2 * i + 1] = v.y;
    }
}

// One whole 32 x 32 block of a tile with 16-bit outputs: two rows at a time, two columns a lane, so
// that an address, a load and a store serve two elements.  csum: the sums of the lane's columns.
template <int kEpi>
__device__ __forceinline__ void block_pairs(const GemmProb &p, int g, int rbase, int nb, const float *tile, int lane,
                                            const float (&av)[32], float2 &csum, float &lsum) {
    const int col = nb + 2 * (lane & 15), row = rbase + (lane >> 4);
    float2 bias = make_float2(0.f, 0.f), wc = make_float2(1.f, 1.f);
    if (kEpi != MCW_EPI_DSILU && p.bias) {
        const float *b = p.bias + (size_t)g * p.s_bias + col;
        bias = make_float2(__ldg(b), __ldg(b + 1));
    }
    if (kEpi == MCW_EPI_LOSS && p.weights) wc = make_float2(__ldg(p.weights + col), __ldg(p.weights + col + 1));
    const float scale = kEpi == MCW_EPI_LOSS ? 1.f / ((float)p.m * (float)p.n) : 0.f;
    __nv_bfloat16 *c16 = static_cast<__nv_bfloat16 *>(p.c) + (size_t)g * p.s_c + (size_t)row * p.ldc + col;
    float *c32 = p.c2 ? p.c2 + (size_t)g * p.s_c2 + (size_t)row * p.ldc2 + col : nullptr;
    const bool has32 = p.c2 != nullptr;
    const float *src = tile + (lane >> 4) * kPitch + 2 * (lane & 15);
    csum = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float2 z = *reinterpret_cast<const float2 *>(src + 2 * i * kPitch);
        if (kEpi != MCW_EPI_DSILU) z.x += bias.x, z.y += bias.y;
        if (kEpi == MCW_EPI_DSILU) z.x *= dsilu(av[2 * i]), z.y *= dsilu(av[2 * i + 1]);
        if (kEpi == MCW_EPI_LOSS) {
            const float dx = z.x - av[2 * i], dy = z.y - av[2 * i + 1];
            lsum += wc.x * dx * dx * scale;
            lsum += wc.y * dy * dy * scale;
            z.x = 2.f * wc.x * dx * scale, z.y = 2.f * wc.y * dy * scale;
        }
        if (kEpi != MCW_EPI_BIAS_SILU) csum.x += z.x, csum.y += z.y;
        if (has32) {
            *reinterpret_cast<float2 *>(c32) = z;
            c32 += 2 * p.ldc2;
        }
        if (kEpi == MCW_EPI_BIAS_SILU) z.x = silu(z.x), z.y = silu(z.y);
        *reinterpret_cast<__nv_bfloat162 *>(c16) = __floats2bfloat162_rn(z.x, z.y);
        c16 += 2 * p.ldc;
    }
    csum.x += __shfl_xor_sync(0xffffffffu, csum.x, 16);
    csum.y += __shfl_xor_sync(0xffffffffu, csum.y, 16);
}

// One 32 x 32 block of a tile, its product in `tile`: a lane's column, row by row.  kFull: the block
// has all its rows and columns.
template <int kEpi, bool kFull>
__device__ __forceinline__ void block_rows(const GemmProb &p, int g, int sp, int rbase, int col, float *tile, int lane,
                                           const float (&av)[32], float &csum, float &lsum) {
    const bool col_ok = kFull || col < p.n;
    const int rows = kFull ? 32 : (col_ok ? min(32, p.m - rbase) : 0);
    float bias = 0.f, wc = 1.f;
    if (kEpi != MCW_EPI_F32 && kEpi != MCW_EPI_DSILU && p.bias && col_ok) bias = __ldg(p.bias + (size_t)g * p.s_bias + col);
    if (kEpi == MCW_EPI_LOSS && p.weights && col_ok) wc = __ldg(p.weights + col);
    const float scale = kEpi == MCW_EPI_LOSS ? 1.f / ((float)p.m * (float)p.n) : 0.f;
    constexpr bool k16 = kEpi == MCW_EPI_BIAS_SILU || kEpi == MCW_EPI_DSILU || kEpi == MCW_EPI_LOSS;
    float *c32 = nullptr;
    long long ld32 = 0;
    __nv_bfloat16 *c16 = nullptr;
    if (!k16) {
        ld32 = p.ldc;
        c32 = static_cast<float *>(p.c) + (size_t)sp * p.s_split + (size_t)g * p.s_c + (size_t)rbase * ld32 + col;
    } else {
        c16 = static_cast<__nv_bfloat16 *>(p.c) + (size_t)g * p.s_c + (size_t)rbase * p.ldc + col;
        ld32 = p.ldc2;
        if (p.c2) c32 = p.c2 + (size_t)g * p.s_c2 + (size_t)rbase * ld32 + col;
    }
    const bool has32 = !k16 || p.c2 != nullptr;
    const bool turned = (kEpi == MCW_EPI_BIAS_SILU || kEpi == MCW_EPI_DSILU) && p.ct;
#pragma unroll
    for (int r = 0; r < 32; ++r) {
        float z = tile[r * kPitch + lane];
        const bool in = kFull || r < rows;
        if (kEpi == MCW_EPI_BIAS_F32 || kEpi == MCW_EPI_BIAS_SILU || kEpi == MCW_EPI_LOSS) z += bias;
        if (kEpi == MCW_EPI_DSILU) z *= dsilu(av[r]);
        if (kEpi == MCW_EPI_LOSS) {
            const float d = z - av[r];
            if (in) lsum += wc * d * d * scale;
            z = 2.f * wc * d * scale;
        }
        if ((kEpi == MCW_EPI_DSILU || kEpi == MCW_EPI_LOSS) && in) csum += z;
        if (has32) {
            if (in) *c32 = z;
            c32 += ld32;
        }
        if (k16) {
            const __nv_bfloat16 h = __float2bfloat16(kEpi == MCW_EPI_BIAS_SILU ? silu(z) : z);
            if (in) *c16 = h;
            c16 += p.ldc;
            if (turned) tile[r * kPitch + lane] = __bfloat162float(h);
        }
    }
    if (turned && col_ok && rows > 0) {
        // transposed copy [n, m]: the lane's column is a run of 32 rows
        __nv_bfloat16 *dst = p.ct + (size_t)g * p.s_ct + (size_t)col * p.ldct + rbase;
        const bool wide = rows == 32 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
        for (int q = 0; q < 4; ++q) {
            uint32_t h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t lo = __float_as_uint(tile[(8 * q + 2 * k) * kPitch + lane]) >> 16;
                h[k] = lo | (__float_as_uint(tile[(8 * q + 2 * k + 1) * kPitch + lane]) & 0xffff0000u);
            }
            if (wide) {
                reinterpret_cast<uint4 *>(dst)[q] = make_uint4(h[0], h[1], h[2], h[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (8 * q + k < rows) dst[8 * q + k] = __ushort_as_bfloat16((unsigned short)(h[k / 2] >> (16 * (k % 2))));
            }
        }
    }
}

// Bias gradients beside weight gradients, 16 columns a CTA behind the tiles' CTAs: the sums of the
// f32 rows colsum_in [k, m] over chunks of colsum_rows rows, rows q, q + 8, ... of a chunk added in
// order for each q < 8 (a thread each), the eight sums in order, the chunks' sums in order
// (mcw_mlp_colsum_grouped's order).  (In the tiles' own epilogue warps, a whole 128 columns fell to
// one CTA of the first layer: 32 us for a launch of 8.)
constexpr int kSumCols = 16;
__device__ __forceinline__ void column_sums(const GemmProb &p, int cta, int tid, float *part) {
    const int tiles = (p.m + kSumCols - 1) / kSumCols;
    const int g = cta / tiles, c = tid % kSumCols, q0 = tid / kSumCols;
    const int col = cta % tiles * kSumCols + c;
    const float *src = p.colsum_in + (size_t)g * p.s_colsum + col;
    float total = 0.f;
    for (int r0 = 0; r0 < p.k; r0 += p.colsum_rows) {
        const int r1 = min(p.k, r0 + p.colsum_rows);
        float s = 0.f;
        if (col < p.m) {
#pragma unroll 16
            for (int r = r0 + q0; r < r1; r += 8) s += __ldg(src + (size_t)r * p.ld_colsum);
        }
        part[tid] = s;
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) t += part[q * kSumCols + c];
        total = r0 == 0 ? t : total + t;
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
    }
    if (q0 == 0 && col < p.m) p.colsum[(size_t)g * p.s_bias + col] = total;
}

template <int kEpi, bool kAMn, bool kBMn, int TN, int kSub>
__global__ void __launch_bounds__(kThreads, 4) gemm_kernel(const __grid_constant__ GemmBatch batch) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], acc_bar;
    __shared__ float part[4 * 32];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    constexpr uint32_t kTmemCols = TN < 32 ? 32 : TN;
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (kAMn ? 1u << 15 : 0u) | (kBMn ? 1u << 16 : 0u) |
                                ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int stages = batch.stages;
    int pi = 0;
    if (kEpi == MCW_EPI_F32 && (int)blockIdx.x >= batch.sums0) {
        while (pi + 1 < batch.np && (int)blockIdx.x >= batch.p[pi + 1].sum0) ++pi;
        after_previous();
        let_next_start();
        if (threadIdx.x < 128) column_sums(batch.p[pi], (int)blockIdx.x - batch.p[pi].sum0, (int)threadIdx.x, part);
        return;
    }
    while (pi + 1 < batch.np && (int)blockIdx.x >= batch.p[pi + 1].cta0) ++pi;
    const GemmProb &p = batch.p[pi];
    int t = (int)blockIdx.x - p.cta0;
    const int n0 = t % p.nt * TN;
    t /= p.nt;
    const int mtile = t % p.mt, m0 = mtile * TM;
    t /= p.mt;
    const int g = t / p.splits, sp = t % p.splits;
    const int kbeg = sp * p.kps;
    const int kend = min(p.k, kbeg + p.kps);
    const int nch = kend > kbeg ? (kend - kbeg + TK - 1) / TK : 0;
    volatile int *abort = &abort_flag;

    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     :: "r"(smem_u32(&tmem_slot)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (threadIdx.x == 128) {
        for (int s = 0; s < stages; ++s) {
            bar_init(&full_bar[s]);
            bar_init(&empty_bar[s]);
        }
        bar_init(&acc_bar);
        asm volatile("fence.mbarrier_init.release.cluster;\n");
        abort_flag = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    const uint32_t ring = smem_u32(smem);
    after_previous();
    let_next_start();

    // K chunks a stage holds, and the stages of this CTA's share
    const int nst = (nch + kSub - 1) / kSub;
    constexpr uint32_t stage = (uint32_t)(kSub * stage_bytes(TN));
    if (warp == 4) {
        int issued = 0;
        bool ready = true;                       // the stage's last use is over
        for (int i = 0, s = 0, use = 0; i < nst; ++i) {
            if (!ready && !warp_wait(&empty_bar[s], (uint32_t)((use - 1) & 1), abort)) break;
            const int s1 = s + 1 == stages ? 0 : s + 1, use1 = s1 == 0 ? use + 1 : use;
            const bool peek = use1 == 0 || test_wait(&empty_bar[s1], (uint32_t)((use1 - 1) & 1));
            const int c0 = i * kSub, cn = kSub == 1 ? 1 : min(kSub, nch - c0);
            if (elect_one()) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n"
                             :: "r"(smem_u32(&full_bar[s])), "r"((uint32_t)(cn * stage_bytes(TN))) : "memory");
#pragma unroll
                for (int c = 0; c < kSub; ++c) {
                    if (c >= cn) break;
                    const uint32_t sa = ring + (uint32_t)s * stage + (uint32_t)(c * stage_bytes(TN));
                    const int k0 = kbeg + (c0 + c) * TK;
                    load_operand<kAMn, TM>(sa, &p.ta, k0, m0, g, &full_bar[s]);
                    load_operand<kBMn, TN>(sa + kABytes, &p.tb, k0, n0, g, &full_bar[s]);
                }
            }
            ready = __all_sync(0xffffffffu, peek);
            issued = i + 1;
            s = s1, use = use1;
        }
        // the last copy into each stage has landed before the CTA can leave
        for (int i = max(0, issued - stages); i < issued; ++i)
            drain_bar(&full_bar[i % stages], (uint32_t)((i / stages) & 1));
    } else if (warp == 5) {
        bool any = false, ready = false;
        for (int i = 0, s = 0, use = 0; i < nst; ++i) {
            if (!ready && !warp_wait(&full_bar[s], (uint32_t)(use & 1), abort)) break;
            // (the next stage is looked at before this one's MMAs are issued, not after)
            const int s1 = s + 1 == stages ? 0 : s + 1, use1 = s1 == 0 ? use + 1 : use;
            const bool peek = i + 1 < nst && test_wait(&full_bar[s1], (uint32_t)(use1 & 1));
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            const int c0 = i * kSub, cn = kSub == 1 ? 1 : min(kSub, nch - c0);
            if (elect_one()) {
#pragma unroll
                for (int c = 0; c < kSub; ++c) {
                    if (c >= cn) break;
                    const uint32_t sa = ring + (uint32_t)s * stage + (uint32_t)(c * stage_bytes(TN));
                    const int steps = (min(TK, kend - kbeg - (c0 + c) * TK) + 15) / 16;
#pragma unroll
                    for (int q = 0; q < TK / 16; ++q) {
                        if (q < steps) {
                            const uint64_t da = operand_desc<kAMn, TM>(sa, q);
                            const uint64_t db = operand_desc<kBMn, TN>(sa + kABytes, q);
                            const uint32_t accumulate = (c0 + c > 0 || q > 0) ? 1u : 0u;
                            asm volatile(
                                "{\n\t.reg .pred p;\n\t"
                                "setp.ne.b32 p, %4, 0;\n\t"
                                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                                :: "r"(tmem), "l"(da), "l"(db), "r"(kIdesc), "r"(accumulate));
                        }
                    }
                }
                commit(&empty_bar[s]);
            }
            ready = __all_sync(0xffffffffu, peek);
            any = true;
            s = s1, use = use1;
        }
        // the accumulator is complete when every MMA issued above is (no MMA: arrives now)
        if (elect_one()) {
            if (any) commit(&acc_bar);
            else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" :: "r"(smem_u32(&acc_bar)) : "memory");
        }
        __syncwarp();
        drain_bar(&acc_bar, 0u);
    } else {
        // the warp's tile lies in the ring, which is free once the accumulator is complete
        float *tile = reinterpret_cast<float *>(smem + (size_t)warp * kTileBytes);
        const int rbase = m0 + warp * 32;
        uint32_t verdict;
        float av[32];
        const bool all_rows = rbase + 32 <= p.m;
        constexpr bool k16 = kEpi == MCW_EPI_BIAS_SILU || kEpi == MCW_EPI_DSILU || kEpi == MCW_EPI_LOSS;
        constexpr bool kAux = kEpi == MCW_EPI_DSILU || kEpi == MCW_EPI_LOSS;
        auto aux_of = [&](int nb) {                   // block nb's other input
            const bool whole = all_rows && nb + 32 <= p.n;
            if (whole && p.pairs) load_aux_pairs(p, g, rbase, nb, lane, av);
            else load_aux(p, g, rbase, nb + lane, whole, av);
        };
        if (kAux) aux_of(n0);
        // the total of the 128-row sums of A's rows, in order
        if (kEpi == MCW_EPI_F32 && p.colsum_in && p.colsum_rows == 0 && sp == 0 && n0 == 0 && rbase + lane < p.m) {
            const float *src = p.colsum_in + (size_t)g * p.s_colsum + rbase + lane;
            float s = 0.f;
            for (int q = 0; q < p.colsum_chunks; ++q) s += src[(size_t)q * p.ld_colsum];
            p.colsum[(size_t)g * p.s_bias + rbase + lane] = s;
        }
        // one verdict for the four warps: they meet at barriers below
        bool ok = wait_bar(&acc_bar, 0u, abort) && !*abort;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "bar.red.and.pred q, 1, 128, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}\n"
            : "=r"(verdict) : "r"(ok ? 1u : 0u) : "memory");
        ok = verdict != 0;
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        float lsum = 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < TN && ok; c0 += 32) {
            const int nb = n0 + c0;
            if (nb >= p.n) break;                                   // block-uniform
            const int col = nb + lane;
            const bool col_ok = col < p.n, whole = all_rows && nb + 32 <= p.n;
            {
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
                __syncwarp();
                float2 *dst = reinterpret_cast<float2 *>(tile + lane * kPitch);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (nch > 0) dst[j] = make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                    else dst[j] = make_float2(0.f, 0.f);
                }
                __syncwarp();
            }
            float csum = 0.f;
            float2 csum2 = make_float2(0.f, 0.f);
            const bool pairs = k16 && whole && p.pairs;
            if constexpr (k16) {
                if (pairs) block_pairs<kEpi>(p, g, rbase, nb, tile, lane, av, csum2, lsum);
            }
            if (!pairs) {
                if (whole) block_rows<kEpi, true>(p, g, sp, rbase, col, tile, lane, av, csum, lsum);
                else block_rows<kEpi, false>(p, g, sp, rbase, col, tile, lane, av, csum, lsum);
            }
            if (kAux) {
                // the next block's other input while this one's sums are put together
                if (c0 + 32 < TN && nb + 32 < p.n) aux_of(nb + 32);
                if (p.colsum) {
                    if (!pairs) part[warp * 32 + lane] = csum;
                    else if (lane < 16) part[warp * 32 + 2 * lane] = csum2.x, part[warp * 32 + 2 * lane + 1] = csum2.y;
                    asm volatile("bar.sync 1, 128;\n" ::: "memory");
                    if (warp == 0 && col_ok)
                        p.colsum[(size_t)g * p.s_colsum + (size_t)mtile * p.ld_colsum + col] =
                            ((part[lane] + part[32 + lane]) + part[64 + lane]) + part[96 + lane];
                    asm volatile("bar.sync 1, 128;\n" ::: "memory");
                }
            }
            __syncwarp();
        }
        if (kEpi == MCW_EPI_LOSS) {
            // one addition to the loss a tile: the sum of many rounds at each
            for (int o = 16; o; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
            if (ok) {
                if (lane == 0) part[warp * 32] = lsum;
                asm volatile("bar.sync 1, 128;\n" ::: "memory");
                if (warp == 0 && lane == 0) atomicAdd(p.loss + g, (part[0] + part[32]) + (part[64] + part[96]));
            }
        }
        if (!ok && lane == 0) atomicOr(batch.err, 4u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    if (warp == 5) {
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" :: "r"(tmem), "r"(kTmemCols));
    }
}

// ---------------------------------------------------------------- host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// The rules of a TMA operand of `inner` contiguous elements per row: 16-byte base, rows and groups
// whole multiples of 16 bytes apart and not overlapping.
bool map_ok(const void *base, long long inner, long long rows, int groups, long long ld, long long stride) {
    return base && !(reinterpret_cast<uintptr_t>(base) & 15) && !(ld & 7) && ld >= inner &&
           (groups == 1 || (!(stride & 7) && stride >= ld * rows));
}

// {inner, rows, groups} bf16 tensor map with a {box_inner, box_rows, 1} box (64 wide: 128-byte
// swizzle, 32 wide: 64-byte).
bool make_map(CUtensorMap *map, const void *base, long long inner, long long rows, int groups, long long ld,
              long long stride, int box_inner, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const long long gstride = groups > 1 ? stride : ld * rows;
    const cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)groups};
    const cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)gstride * 2};
    const cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE,
              box_inner == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int kEpi, bool kAMn, bool kBMn, int TN, int kSub = 1>
cudaError_t launch(const GemmBatch &b, unsigned grid, size_t smem, cudaStream_t s) {
    auto *kernel = gemm_kernel<kEpi, kAMn, kBMn, TN, kSub>;
    const cudaError_t e = allow_smem(reinterpret_cast<const void *>(kernel), 208 * 1024);
    if (e != cudaSuccess) return e;
    return launch_after(kernel, grid, kThreads, smem, s, b);
}

// The combinations of epilogue and layouts that exist: a plain product takes any, a backward
// product a transposed B (the weights), the others rows along K.
bool has_kernel(int epi, bool ta, bool tb) {
    return epi == MCW_EPI_F32 || (!ta && (!tb || epi == MCW_EPI_DSILU));
}

template <int TN>
cudaError_t launch_n(int epi, const GemmBatch &b, bool ta, bool tb, unsigned grid, size_t smem, cudaStream_t s) {
    switch (epi) {
        case MCW_EPI_F32:
            if constexpr (TN == 32) {              // (tiles of 64 columns: more than an SM's, the rule in launch_batch)
                if (ta && tb && b.sub == 2) return launch<MCW_EPI_F32, true, true, TN, 2>(b, grid, smem, s);
            }
            if (ta) return tb ? launch<MCW_EPI_F32, true, true, TN>(b, grid, smem, s)
                              : launch<MCW_EPI_F32, true, false, TN>(b, grid, smem, s);
            return tb ? launch<MCW_EPI_F32, false, true, TN>(b, grid, smem, s)
                      : launch<MCW_EPI_F32, false, false, TN>(b, grid, smem, s);
        case MCW_EPI_BIAS_F32: return launch<MCW_EPI_BIAS_F32, false, false, TN>(b, grid, smem, s);
        case MCW_EPI_BIAS_SILU: return launch<MCW_EPI_BIAS_SILU, false, false, TN>(b, grid, smem, s);
        case MCW_EPI_DSILU:
            return tb ? launch<MCW_EPI_DSILU, false, true, TN>(b, grid, smem, s)
                      : launch<MCW_EPI_DSILU, false, false, TN>(b, grid, smem, s);
        default: return launch<MCW_EPI_LOSS, false, false, TN>(b, grid, smem, s);
    }
}

long long tiles_of(const McwGemmProblem &q, int tn, int splits) {
    return (long long)((q.m + TM - 1) / TM) * ((q.n + tn - 1) / tn) * q.groups * splits;
}

// Checked problems in one launch.
int launch_batch(const McwGemmProblem *q, int np, cudaStream_t stream) {
    static thread_local GemmBatch b;
    memset(&b, 0, sizeof(b));
    b.np = np;
    b.err = tc_err_flag();
    if (!b.err) return MCW_MLP_ERR_CUDA;
    const bool ta = q[0].trans_a != 0, tb = q[0].trans_b != 0;
    long long t64 = 0, t32 = 0;
    int chunks = 1;
    for (int i = 0; i < np; ++i) {
        t64 += tiles_of(q[i], 64, q[i].splits);
        t32 += tiles_of(q[i], 32, q[i].splits);
        const int c = ((q[i].k + TK - 1) / TK + q[i].splits - 1) / q[i].splits;
        chunks = c > chunks ? c : chunks;
    }
    const int sms = sm_count();
    // 64 columns a tile when that leaves two tiles per SM: at 65,536 rows with tiles of 32 / 64
    // columns the SiLU' product of 649 takes 92 / 69 us, of 256 62 / 51 (bias + SiLU 256 x 256 53 / 36,
    // the 256 x 649 output 84 / 72)
    const int tn = t64 >= 2 * sms ? 64 : 32;
    // two stages when the launch fills the SMs several times over (four CTAs of an SM overlap each
    // other), else up to eight, or as many as the chunks; five of two chunks each for a transposed
    // product with an SM to a CTA and a long chain, where a stage's handover (120 ns beside 20 ns an
    // MMA) is what is left: the weight gradients of 65,536 rows, 1,024 chunks a tile, take
    // 464 / 317 / 246 / 201 us with 2 / 3 / 4 / 8 stages, 176 with 5 of two
    const long long ctas = tn == 64 ? t64 : t32;
    const int stages = ctas > 2 * sms ? 2 : (ctas > sms ? 4 : kMaxStages);
    b.stages = stages > chunks ? chunks : stages;
    b.sub = q[0].epilogue == MCW_EPI_F32 && ta && tb && ctas <= sms && chunks >= 4 * kMaxStages ? 2 : 1;
    if (b.sub == 2) b.stages = 5;
    long long cta = 0;
    for (int i = 0; i < np; ++i) {
        const McwGemmProblem &s = q[i];
        GemmProb &d = b.p[i];
        const int wide = tn < 64 ? 32 : 64;
        if (!(s.trans_a ? make_map(&d.ta, s.a, s.m, s.k, s.groups, s.lda, s.stride_a, 64, 64)
                        : make_map(&d.ta, s.a, s.k, s.m, s.groups, s.lda, s.stride_a, 64, TM)))
            return MCW_MLP_ERR_ARG;
        if (!(s.trans_b ? make_map(&d.tb, s.b, s.n, s.k, s.groups, s.ldb, s.stride_b, wide, 64)
                        : make_map(&d.tb, s.b, s.k, s.n, s.groups, s.ldb, s.stride_b, 64, tn)))
            return MCW_MLP_ERR_ARG;
        d.m = s.m, d.n = s.n, d.k = s.k;
        d.mt = (s.m + TM - 1) / TM;
        d.nt = (s.n + tn - 1) / tn;
        const int ch = (s.k + TK - 1) / TK;
        d.splits = s.splits;
        d.kps = (ch + s.splits - 1) / s.splits * TK;
        d.cta0 = (int32_t)cta;
        cta += tiles_of(s, tn, s.splits);
        d.bias = s.bias, d.s_bias = s.stride_bias;
        d.aux = s.aux, d.ld_aux = s.ldaux, d.s_aux = s.stride_aux;
        d.c = s.c, d.ldc = s.ldc, d.s_c = s.stride_c, d.s_split = s.stride_split;
        d.c2 = static_cast<float *>(s.c2), d.ldc2 = s.ldc2, d.s_c2 = s.stride_c2;
        d.ct = static_cast<__nv_bfloat16 *>(s.ct), d.ldct = s.ldct, d.s_ct = s.stride_ct;
        d.colsum = s.colsum, d.colsum_in = s.colsum_in, d.s_colsum = s.stride_colsum, d.ld_colsum = s.ld_colsum;
        d.colsum_chunks = s.colsum_chunks, d.colsum_rows = s.colsum_rows;
        d.weights = s.weights, d.loss = s.loss;
        auto even = [](const void *p, long long ld, long long stride, int bytes) {
            return !p || (!(reinterpret_cast<uintptr_t>(p) % (2 * bytes)) && !(ld & 1) && !(stride & 1));
        };
        d.pairs = (s.epilogue == MCW_EPI_BIAS_SILU || s.epilogue == MCW_EPI_DSILU || s.epilogue == MCW_EPI_LOSS) && !s.ct &&
                  even(s.c, s.ldc, s.stride_c, 2) && even(s.c2, s.ldc2, s.stride_c2, 4) && even(s.aux, s.ldaux, s.stride_aux, 4);
    }
    b.sums0 = cta > 0x7fffffffLL ? 0 : (int32_t)cta;
    for (int i = 0; i < np; ++i) {
        b.p[i].sum0 = (int32_t)cta;
        if (q[i].epilogue == MCW_EPI_F32 && q[i].colsum_in && q[i].colsum_rows > 0)
            cta += (long long)((q[i].m + kSumCols - 1) / kSumCols) * q[i].groups;
    }
    if (cta > 0x7fffffffLL) return MCW_MLP_ERR_ARG;
    const size_t ring = (size_t)b.stages * b.sub * stage_bytes(tn), tiles = 4 * kTileBytes;
    const size_t smem = (ring > tiles ? ring : tiles) + 1024;
    cudaError_t e;
    if (tn == 64) e = launch_n<64>(q[0].epilogue, b, ta, tb, (unsigned)cta, smem, stream);
    else e = launch_n<32>(q[0].epilogue, b, ta, tb, (unsigned)cta, smem, stream);
    return e == cudaSuccess ? 0 : MCW_MLP_ERR_CUDA;
}

bool operands_ok(const McwGemmProblem &s) {
    return (s.trans_a ? map_ok(s.a, s.m, s.k, s.groups, s.lda, s.stride_a)
                      : map_ok(s.a, s.k, s.m, s.groups, s.lda, s.stride_a)) &&
           (s.trans_b ? map_ok(s.b, s.n, s.k, s.groups, s.ldb, s.stride_b)
                      : map_ok(s.b, s.k, s.n, s.groups, s.ldb, s.stride_b));
}

}  // namespace

// mcw_mlp_gemm on this kernel: false when an operand breaks the copies' rules (the caller then
// stages it by threads).
bool gemm_by_tma(const McwGemm &p, cudaStream_t s, int *rc) {
    McwGemmProblem q;
    memset(&q, 0, sizeof(q));
    q.m = p.m, q.n = p.n, q.k = p.k, q.groups = 1, q.splits = 1, q.epilogue = p.epilogue;
    q.trans_a = p.trans_a ? 1 : 0, q.trans_b = p.trans_b ? 1 : 0;
    q.a = p.a, q.lda = p.lda, q.b = p.b, q.ldb = p.ldb;
    q.bias = p.bias, q.aux = p.aux, q.ldaux = p.ldaux, q.c = p.c, q.ldc = p.ldc, q.c2 = p.c2, q.ldc2 = p.ldc2;
    if (p.epilogue > MCW_EPI_DSILU || !has_kernel(p.epilogue, q.trans_a, q.trans_b) || p.k <= 0 || !operands_ok(q))
        return false;
    if (p.epilogue == MCW_EPI_F32 || p.epilogue == MCW_EPI_BIAS_F32) q.c2 = nullptr;
    *rc = launch_batch(&q, 1, s);
    return true;
}

}  // namespace mcw

using namespace mcw;

extern "C" {

int mcw_mlp_gemm_batch(const McwGemmProblem *q, int32_t n, void *stream) {
    if (!q || n < 1 || n > MCW_GEMM_BATCH_MAX) return MCW_MLP_ERR_ARG;
    McwGemmProblem kept[MCW_GEMM_BATCH_MAX];
    int np = 0;
    for (int i = 0; i < n; ++i) {
        const McwGemmProblem &s = q[i];
        if (s.m < 0 || s.n < 0 || s.k <= 0 || s.groups < 1 || s.splits < 1 || !s.a || !s.b || !s.c) return MCW_MLP_ERR_ARG;
        if (s.m == 0 || s.n == 0) continue;                   // nothing to do, whatever the rest
        if (s.epilogue < MCW_EPI_F32 || s.epilogue > MCW_EPI_LOSS) return MCW_MLP_ERR_ARG;
        if (np > 0 && (s.epilogue != kept[0].epilogue || (s.trans_a != 0) != (kept[0].trans_a != 0) ||
                       (s.trans_b != 0) != (kept[0].trans_b != 0)))
            return MCW_MLP_ERR_ARG;
        if (!has_kernel(s.epilogue, s.trans_a != 0, s.trans_b != 0)) return MCW_MLP_ERR_ARG;
        if (s.splits > 1 && s.epilogue != MCW_EPI_F32) return MCW_MLP_ERR_ARG;
        if (s.epilogue == MCW_EPI_BIAS_SILU && !s.bias) return MCW_MLP_ERR_ARG;
        if ((s.epilogue == MCW_EPI_DSILU || s.epilogue == MCW_EPI_LOSS) && !s.aux) return MCW_MLP_ERR_ARG;
        if (s.epilogue == MCW_EPI_LOSS && (!s.loss || !s.bias)) return MCW_MLP_ERR_ARG;
        if (s.epilogue == MCW_EPI_F32 && s.colsum_in && (!s.colsum || s.colsum_chunks < 0 || s.colsum_rows < 0))
            return MCW_MLP_ERR_ARG;
        if ((long long)s.groups * s.splits > 65535) return MCW_MLP_ERR_ARG;
        const int chunks = (s.k + TK - 1) / TK;
        const int per = (chunks + s.splits - 1) / s.splits;
        if (s.splits > 1 && (chunks + per - 1) / per != s.splits) return MCW_MLP_ERR_ARG;   // the caller's partial layout
        if (!operands_ok(s)) return MCW_MLP_ERR_ARG;
        kept[np++] = s;
    }
    return np ? launch_batch(kept, np, static_cast<cudaStream_t>(stream)) : 0;
}

int mcw_mlp_gemm_grouped(const McwGemmGrouped *q, void *stream) {
    if (!q) return MCW_MLP_ERR_ARG;
    if (q->epilogue > MCW_EPI_DSILU && q->m != 0 && q->n != 0) return MCW_MLP_ERR_ARG;
    McwGemmProblem s;
    memset(&s, 0, sizeof(s));
    s.m = q->m, s.n = q->n, s.k = q->k, s.groups = q->groups, s.splits = q->splits, s.epilogue = q->epilogue;
    s.a = q->a, s.lda = q->lda, s.stride_a = q->stride_a;
    s.b = q->b, s.ldb = q->ldb, s.stride_b = q->stride_b;
    s.bias = q->bias, s.stride_bias = q->stride_bias;
    s.aux = q->aux, s.ldaux = q->ldaux, s.stride_aux = q->stride_aux;
    s.c = q->c, s.ldc = q->ldc, s.stride_c = q->stride_c, s.stride_split = q->stride_split;
    s.c2 = q->c2, s.ldc2 = q->ldc2, s.stride_c2 = q->stride_c2;
    s.ct = q->ct, s.ldct = q->ldct, s.stride_ct = q->stride_ct;
    return mcw_mlp_gemm_batch(&s, 1, stream);
}

}  // extern "C"
