"""CPU: the host-side rules that choose the eikonal solver's kernel (csrc/fim.cuh), compiled from
the header itself: which launch errors mean that a device has no place for a cluster (all others
are reported, not worked around)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "seismic_tomography_3d_b200", "csrc")
SRC = r"""
#include <cstdio>
#include "fim.cuh"
using namespace tomo;
#define CHECK(x) do { if (!(x)) { printf("%s\n", #x); return 1; } } while (0)
int main()
{
    for (cudaError_t e : {cudaErrorInvalidClusterSize, cudaErrorLaunchOutOfResources, cudaErrorInvalidConfiguration,
                          cudaErrorNotSupported})
        CHECK(no_place_for_cluster(e));
    for (cudaError_t e : {cudaSuccess, cudaErrorInvalidValue, cudaErrorMemoryAllocation, cudaErrorInvalidDeviceFunction,
                          cudaErrorIllegalAddress, cudaErrorLaunchFailure, cudaErrorStreamCaptureInvalidated, cudaErrorUnknown})
        CHECK(!no_place_for_cluster(e));
    return 0;
}
"""


def test_rules(tmp_path):
    (tmp_path / "d.cpp").write_text(SRC)
    exe = str(tmp_path / "d")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, "-I" + os.path.join(cuda, "include"), "-o", exe,
                    str(tmp_path / "d.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
