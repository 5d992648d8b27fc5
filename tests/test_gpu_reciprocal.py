"""The branchless reciprocal of the activations (fk_recip.cuh) against the division, for every float that it is used for."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include "fk_recip.cuh"
__global__ void look(uint32_t from, uint32_t to, unsigned long long *bad) {
    unsigned long long n = 0;
    for (unsigned long long i = from + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < to; i += (unsigned long long)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((uint32_t)i);
        n += __float_as_uint(recip_from_one(x)) != __float_as_uint(__fdiv_rn(1.0f, x));
    }
    if (n) atomicAdd(bad, n);
}
int main() {
    const float a = 1.0f, b = FK_RECIP_END;
    uint32_t from, to;
    memcpy(&from, &a, 4); memcpy(&to, &b, 4);
    unsigned long long *bad, n = 0;
    if (cudaMalloc(&bad, 8) != cudaSuccess || cudaMemset(bad, 0, 8) != cudaSuccess) return 1;
    look<<<1184, 256>>>(from, to, bad);
    if (cudaMemcpy(&n, bad, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("%u floats, %llu differ\n", to - from, n);
    return 0;
}
"""


def test_every_float_from_one_on(tmp_path):
    (tmp_path / "look.cu").write_text(PROGRAM)
    exe = str(tmp_path / "look")
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-include", "cstring", "-I", os.path.join(ROOT, "fusekit_b200", "csrc"), "-o", exe,
                           str(tmp_path / "look.cu")])
    out = subprocess.check_output([exe], text=True, timeout=120)
    assert out == f"{126 << 23} floats, 0 differ\n", out
