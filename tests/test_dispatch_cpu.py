"""CPU: the host-side rules that choose the eikonal solver's kernel (csrc/fim.cuh), compiled from
the header itself: which launch errors mean that a device has no place for a cluster (all others
are reported, not worked around), and when the one-brick kernel runs one CTA per SM: on the side of
every measured pair that was faster."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "seismic_tomography_3d_b200", "csrc")
SRC = r"""
#include <cmath>
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
    struct { int shots; unsigned long long bricks; int ctas; } measured[] = {
        {1, 67626, 1}, {2, 67626, 1}, {10, 8788, 1}, {12, 8788, 1}, {5, 792, 1}, {30, 792, 1}, {64, 75, 1},
        {1, 256000, 0}, {1, 320000, 0}, {15, 8788, 0}, {18, 8788, 0}, {24, 8788, 0}, {10, 15750, 0}, {400, 75, 0}};
    for (const auto &m : measured)
        CHECK(rounds_ctas_per_sm(false, m.shots * m.bricks, m.shots * std::pow((double)m.bricks, 2.0 / 3.0)) == m.ctas);
    CHECK(rounds_ctas_per_sm(true, 75, std::pow(75.0, 2.0 / 3.0)) == 0);  // a chosen shape is kept
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
