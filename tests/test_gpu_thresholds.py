"""The acceptance threshold of a random word as the sweep kernels compute it (word_threshold and
neglog_quotient, csrc/rng.cuh) against the general routine and CUDA's correctly rounded division,
for every word the generator can produce that matters (the lowest bit does not: 2^31 of them)."""
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "rng.cuh"
using namespace rewl;
__global__ void compare(unsigned long long* bad)
{
    const uint32_t v = 2u * (blockIdx.x * blockDim.x + threadIdx.x) + 1u;
    const bool high = v > 0xB504F333u;
    const int e = 31 - __clz(v);
    const float d = __fmul_rn(__uint2float_rn(0u - v), 2.3283064365386963e-10f);
    float m = __fmul_rn(__uint2float_rn(v), __uint_as_float((uint32_t)(127 - e) << 23));
    if (m > 1.41421354f) m = __fmul_rn(m, 0.5f);
    const float num = high ? d : __fsub_rn(1.0f, m), den = high ? __fsub_rn(2.0f, d) : __fadd_rn(m, 1.0f);
    if (neglog_quotient(num, den) != __fdiv_rn(num, den)) atomicAdd(bad, 1ull);
    if (word_threshold(v) != accept_threshold(neglog_u32(v))) atomicAdd(bad + 1, 1ull);
}
int main()
{
    unsigned long long *b, h[2] = {1, 1};
    if (cudaMalloc(&b, sizeof h) != cudaSuccess || cudaMemset(b, 0, sizeof h) != cudaSuccess) return 2;
    compare<<<1u << 23, 256>>>(b);
    if (cudaMemcpy(h, b, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("%llu %llu\n", h[0], h[1]);
    return 0;
}
"""


@pytest.mark.gpu
def test_every_word(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "compare.cu").write_text(PROGRAM)
    exe = tmp_path / "compare"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-I", str(ROOT / "rewl_simulator_gb300" / "csrc"), str(tmp_path / "compare.cu"), "-o", str(exe)],
                   check=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, timeout=120, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0"], out
