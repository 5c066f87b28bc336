"""Square roots and quotients of the FP64 replay and the FP32 reciprocal of SiLU's derivative
(csrc/rounded.cuh) against IEEE arithmetic, bit for bit: arguments whose exact result lies next to the
middle between two doubles, where the kernels' correction alone rounds to the wrong side, arguments at
random, zeros, infinities, NaN, denormals and powers of two; every float from 1 on."""
import ctypes
import subprocess

import numpy as np
import pytest

from monte_carlompi_gb300 import build

pytestmark = pytest.mark.gpu

PROBE = r'''
#include "rounded.cuh"
using namespace mcw;
__global__ void probe(const double *a, const double *b, int n, double *q, double *s, unsigned char *wrong) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double h;
    const double rb = rcp_res(b[i]), g = sqrt_res(b[i], h), r = quotient_res(a[i], b[i], rb);
    q[i] = quotient_sure(r, a[i], b[i]) ? r : a[i] / b[i];
    s[i] = sqrt_sure(g, b[i]) ? g : sqrt(b[i]);
    // 1, 2: the root, the quotient by its doubled reciprocal certain; 4: the corrections alone, not as sqrt or /
    const bool pos = b[i] > 0 && moderate(b[i]);
    wrong[i] = (pos && sqrt_certain(g, b[i]) ? 1 : 0) | (moderate(b[i]) && quotient_certain(r, a[i], b[i]) ? 2 : 0) |
               (pos && g != sqrt(b[i]) ? 4 : 0) | (moderate(b[i]) && r != a[i] / b[i] ? 8 : 0);
}
__global__ void reciprocals(unsigned *bad) {
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = 0x3f800000ull + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i <= 0x7fc00000ull; i += step) {
        const float d = __uint_as_float((unsigned)i), s = reciprocal_rn(d), want = 1.f / d;
        if (s != want && !(s != s && want != want)) atomicAdd(bad, 1u);
    }
}
// How many floats from 1 to infinity, and NaN, have another reciprocal than 1.f / d.
extern "C" int reciprocals_off(unsigned *off) {
    unsigned *d = nullptr;
    if (cudaMalloc(&d, 4)) return 1;
    cudaMemset(d, 0, 4);
    reciprocals<<<1216, 256>>>(d);
    cudaMemcpy(off, d, 4, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)cudaGetLastError();
}
extern "C" int run(const double *a, const double *b, int n, double *q, double *s, unsigned char *wrong) {
    double *d = nullptr;
    unsigned char *w = nullptr;
    if (cudaMalloc(&d, (size_t)n * 32) || cudaMalloc(&w, n)) return 1;
    cudaMemcpy(d, a, (size_t)n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, (size_t)n * 8, cudaMemcpyHostToDevice);
    probe<<<(n + 255) / 256, 256>>>(d, d + n, n, d + 2 * (size_t)n, d + 3 * (size_t)n, w);
    cudaMemcpy(q, d + 2 * (size_t)n, (size_t)n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(s, d + 3 * (size_t)n, (size_t)n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(wrong, w, n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(w);
    return (int)cudaGetLastError();
}
'''


@pytest.fixture(scope='module')
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp('rounded')
    (d / 'probe.cu').write_text(PROBE)
    subprocess.run([build.nvcc(), *build.ARCH, '-O3', '-std=c++17', '--fmad=false', '-I', build.CSRC, '-shared', '-Xcompiler',
                    '-fPIC', str(d / 'probe.cu'), '-o', str(d / 'probe.so')], check=True)
    lib = ctypes.CDLL(str(d / 'probe.so'))

    def run(a, b):
        a, b = (np.ascontiguousarray(np.broadcast_to(t, np.broadcast_shapes(np.shape(a), np.shape(b))), np.float64).ravel()
                for t in (a, b))
        q, s, w = np.empty_like(a), np.empty_like(a), np.empty(a.size, np.uint8)
        p = lambda t: ctypes.c_void_p(t.ctypes.data)  # noqa: E731
        assert lib.run(p(a), p(b), a.size, p(q), p(s), p(w)) == 0
        with np.errstate(all='ignore'):
            return a, b, q, a / b, s, np.sqrt(b), w
    run.lib = lib
    return run


def same(got, want):
    return np.where(np.isnan(want), np.isnan(got), got.view(np.uint64) == want.view(np.uint64)).all()


def hard_roots(count):
    """x in (0, 1] whose square roots lie within 2^-40 ulp of a middle: (odd n)^2 = X 2^s + c."""
    out = []
    for c in range(1, count * 8, 8):
        for c_ in (c, c - 8 * count):
            for s in (54, 55):
                r = 1
                for k in range(3, s):                      # r^2 = c modulo 2^(k + 1)
                    if (r * r - c_) >> k & 1:
                        r += 1 << (k - 1)
                for n in {t % (1 << s) for t in (r, -r, r + (1 << (s - 1)), -r - (1 << (s - 1)))}:
                    x = (n * n - c_) >> s
                    if (n * n - c_) == x << s and x.bit_length() == 53 and n.bit_length() == 54:
                        out.append(float(x) * 2.0 ** (s - 108))
    return np.array(out)


def hard_quotients(rng, count):
    """a, b in [1, 2) with a / b next to a middle: (odd n) b = a 2^s + c."""
    a, b = [], []
    while len(a) < count:
        bi = int(rng.integers(1 << 52, 1 << 53)) | 1
        for c in (1, -1, 3, -5):
            for s in (53, 54):
                n = c * pow(bi, -1, 1 << s) % (1 << s)
                n += 1 << 53 if s == 53 else 0
                ai = (n * bi - c) >> s
                if n.bit_length() == 54 and ai.bit_length() == 53:
                    a.append(float(ai) * 2.0 ** -52)
                    b.append(float(bi) * 2.0 ** -52)
    return np.array(a), np.array(b)


def test_next_to_the_middle_of_two_doubles(probe):
    x = hard_roots(2000)
    assert x.size > 2000 and (x <= 1).all()
    _, _, _, _, s, want, w = probe(1.0, np.concatenate([x, x * 2.0 ** -40]))
    assert same(s, want)
    assert not (w & 1).any() and (w & 4).mean() > 0.1      # none taken for certain; many were wrong
    a, b = hard_quotients(np.random.default_rng(1), 20000)
    for fa, fb in ((1, 1), (-2.0 ** -30, 2.0 ** -20), (2.0 ** -300, 1), (1, 2.0 ** -200)):
        _, _, q, want, _, _, w = probe(a * fa, b * fb)
        assert same(q, want) and not (w & 2).any() and (w & 8).mean() > 0.1


def test_at_random_and_at_the_ends(probe):
    rng = np.random.default_rng(2)
    b = 2.0 ** rng.uniform(-52, 0, 1 << 22)
    a, b, q, qw, s, sw, w = probe(rng.standard_normal(b.size) * 2.0 ** rng.integers(-60, 60, b.size), b)
    assert same(q, qw) and same(s, sw)
    assert not (((w & 1) > 0) & ((w & 4) > 0)).any() and not (((w & 2) > 0) & ((w & 8) > 0)).any()
    assert ((w & 3) != 3).mean() < 1e-4                    # (most results are certain)
    ends = np.array([0.0, 1.0, 1 - 2.0 ** -53, 2.0 ** -53, 1 + 2.0 ** -52, 2.0, 3.0, 2.0 ** 52, 2.0 ** 53, 2.0 ** 1023, 5e-324,
                     2.0 ** -1022, 2.0 ** -255, 2.0 ** -256, 2.0 ** -1000, 1e300, np.inf, np.nan, 0.1, 1.7976931348623157e308])
    ends = np.concatenate([ends, -ends])
    _, _, q, qw, s, sw, _ = probe(ends[:, None], ends[None, :])
    assert same(q, qw) and same(s, sw)


def test_every_reciprocal_from_one_on(probe):
    off = ctypes.c_uint32(1)
    assert probe.lib.reciprocals_off(ctypes.byref(off)) == 0 and off.value == 0
