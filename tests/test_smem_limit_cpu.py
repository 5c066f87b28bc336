"""The shared-memory limit of the library's kernels (csrc/smem_limit.cuh), on a CUDA runtime of the
test's own: asked of every device and kernel once, again when more is wanted and after a failure."""
import glob
import os
import re
import subprocess

from monte_carlompi_gb300 import build

CHECK = r'''
#include <cassert>
#include "smem_limit.cuh"
static int device = 0, asked = 0;
static cudaError_t answer = cudaSuccess;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { ++asked; return answer; }
int main() {
    int a, b;
    using mcw::allow_smem;
    answer = cudaErrorInvalidValue;
    if (allow_smem(&a, 100) == cudaSuccess || asked != 1) return 1;
    answer = cudaSuccess;
    if (allow_smem(&a, 100) != cudaSuccess || asked != 2) return 2;   // not remembered as failed
    if (allow_smem(&a, 100) != cudaSuccess || allow_smem(&a, 50) != cudaSuccess || asked != 2) return 3;
    if (allow_smem(&b, 100) != cudaSuccess || asked != 3) return 4;
    if (allow_smem(&a, 200) != cudaSuccess || asked != 4) return 5;
    device = 1;
    if (allow_smem(&a, 200) != cudaSuccess || asked != 5) return 6;   // the other device's own
    device = 0;
    if (allow_smem(&a, 200) != cudaSuccess || asked != 5) return 7;
    return 0;
}
'''


def test_limit_is_asked_per_device_and_kernel(tmp_path):
    src, exe = tmp_path / 'check.cpp', tmp_path / 'check'
    src.write_text(CHECK)
    include = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), 'include')
    subprocess.run([os.environ.get('CXX', 'g++'), '-std=c++17', '-I', build.CSRC, '-I', include, str(src), '-o', str(exe),
                    '-lpthread'], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_kernel_attribute_is_set_once_per_process():
    for path in glob.glob(os.path.join(build.CSRC, '*.cu*')):
        for body in re.findall(r'call_once\((.*?)\}\);', open(path).read(), re.S):
            assert 'cudaFuncSetAttribute' not in body, path
