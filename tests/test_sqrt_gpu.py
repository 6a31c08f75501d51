"""fsqrt of csrc/common.cuh against the IEEE square root, for every float it is exact for
([2^-102, 2^126)), and its zero, infinity and negative arguments, in a small program built
from the header itself."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "seismic_tomography_3d_b200", "csrc")
SRC = r"""
#include <cmath>
#include <cstdio>
#include "common.cuh"
__global__ void every(unsigned lo, unsigned hi, unsigned long long *bad)
{
    unsigned long long n = 0;
    for (unsigned long long u = lo + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; u < hi;
         u += gridDim.x * (unsigned long long)blockDim.x) {
        const float a = __uint_as_float((unsigned)u);
        n += tomo::fsqrt(a) != __fsqrt_rn(a);
    }
    atomicAdd(bad, n);
}
__global__ void some(const float *a, float *s, int n) { if (threadIdx.x < n) s[threadIdx.x] = tomo::fsqrt(a[threadIdx.x]); }
int main()
{
    unsigned long long *bad, n = 1;
    float *d, h[4] = {0.0f, -0.0f, -1.0f, -1e-30f};
    if (cudaMalloc(&bad, sizeof(n)) || cudaMemset(bad, 0, sizeof(n)) || cudaMalloc(&d, 8 * sizeof(float))) return 2;
    every<<<148 * 8, 256>>>((127u - 102u) << 23, (127u + 126u) << 23, bad);
    cudaMemcpy(d, h, sizeof(h), cudaMemcpyHostToDevice);
    some<<<1, 32>>>(d, d + 4, 4);
    if (cudaMemcpy(&n, bad, sizeof(n), cudaMemcpyDeviceToHost) || cudaMemcpy(h, d + 4, sizeof(h), cudaMemcpyDeviceToHost)) return 2;
    printf("%llu wrong, %g %g %g %g\n", n, h[0], h[1], h[2], h[3]);
    return n || h[0] != 0.0f || h[1] != 0.0f || h[2] == h[2] || h[3] == h[3];
}
"""


def test_every_root(tmp_path):
    (tmp_path / "s.cu").write_text(SRC)
    exe = str(tmp_path / "s")
    subprocess.run([os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc"), "-gencode",
                    "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I" + CSRC, "-o", exe, str(tmp_path / "s.cu")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
