"""rsqrt_normal and log2_normal against rsqrtf and __log2f: the same bits for
every argument that is not subnormal (both zeros, infinities, NaN and negative
numbers among them), over all FP32 numbers."""
import os
import subprocess

import pytest

from gravity_gb300 import build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "gbh_common.cuh"
__device__ bool differ(float a, float b) {
    return __float_as_uint(a) != __float_as_uint(b) && !(isnan(a) && isnan(b));
}
__global__ void k_compare(unsigned long long* bad) {
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < 1ull << 32; i += stride) {
        const uint32_t u = (uint32_t)i;
        if ((u & 0x7F800000u) == 0u && (u & 0x007FFFFFu)) continue;  // subnormal
        const float x = __uint_as_float(u);
        if (differ(rsqrt_normal(x), rsqrtf(x))) atomicAdd(bad, 1ull);
        if (differ(log2_normal(x), __log2f(x))) atomicAdd(bad + 1, 1ull);
    }
}
int main() {
    unsigned long long* bad;
    unsigned long long host[2] = {1, 1};
    if (cudaMalloc(&bad, 16) != cudaSuccess || cudaMemset(bad, 0, 16) != cudaSuccess) return 2;
    k_compare<<<1024, 256>>>(bad);
    if (cudaMemcpy(host, bad, 16, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    printf("%llu %llu\n", host[0], host[1]);
    return 0;
}
"""


def test_one_instruction_forms_give_the_functions_bits(tmp_path):
    src, exe = tmp_path / "compare.cu", tmp_path / "compare"
    src.write_text(PROGRAM)
    nvcc = os.environ.get("NVCC", "nvcc")
    r = subprocess.run([nvcc] + build.FLAGS + ["--fmad=false", "-I", build.CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["0", "0"]
