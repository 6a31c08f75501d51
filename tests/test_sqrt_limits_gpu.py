"""fsqrt of csrc/common.cuh outside the range in which it is exact: NaN for subnormal and for
infinite arguments, as its comment says, so its callers have to keep them out."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "seismic_tomography_3d_b200", "csrc")
SRC = r"""
#include <cstdio>
#include "common.cuh"
__global__ void roots(const float *a, float *s) { s[threadIdx.x] = tomo::fsqrt(a[threadIdx.x]); }
int main()
{
    float *d, h[4] = {0x1p-149f, 0x1.fffffcp-127f, 1e38f * 10.0f, -1e38f * 10.0f};
    if (cudaMalloc(&d, 8 * sizeof(float)) || cudaMemcpy(d, h, sizeof(h), cudaMemcpyHostToDevice)) return 2;
    roots<<<1, 4>>>(d, d + 4);
    if (cudaMemcpy(h, d + 4, sizeof(h), cudaMemcpyDeviceToHost)) return 2;
    printf("%g %g %g %g\n", h[0], h[1], h[2], h[3]);
    return h[0] == h[0] || h[1] == h[1] || h[2] == h[2] || h[3] == h[3];
}
"""


def test_outside_the_range(tmp_path):
    (tmp_path / "s.cu").write_text(SRC)
    exe = str(tmp_path / "s")
    subprocess.run([os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc"), "-gencode",
                    "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I" + CSRC, "-o", exe, str(tmp_path / "s.cu")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
