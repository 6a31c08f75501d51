"""CPU: the choice between 32- and 64-bit field offsets in the ray march (csrc/ray.cuh).  The
largest field marched in 32 bits must have all its offsets below 2^31, and the choice is part of
the geometry that a captured iteration is keyed by (JacGeom): windows may grow past 2^31 nodes
while counts, buffers and everything else of the key stay."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "seismic_tomography_3d_b200", "csrc")
SRC = r"""
#include <cstdio>
#include <cstring>
#include "internal.hpp"
using namespace tomo;
static ShotDesc field(int bx, int by, int bz) { ShotDesc d{}; d.nbx = bx; d.nby = by; d.nbz = bz; return d; }
// the march's offset of a node: the sum of one part per axis, in the type chosen
static long long offset(const ShotDesc &d, int x, int y, int z)
{
    const long long sx = 64ll * d.nbz - 16, sy = 64ll * d.nbz * d.nbx - 64;
    return z + 60ll * (z >> 2) + 4ll * x + sx * (x >> 2) + 16ll * y + sy * (y >> 2);
}
int main()
{
    const ShotDesc narrow = field(511, 1024, 64), odd = field(3, 5592405, 2), edge = field(512, 1024, 64), big = field(2048, 2048, 512);
    ShotDesc two[2] = {narrow, big};
    if (wide_fields(&narrow, 1) || wide_fields(&odd, 1) || !wide_fields(&edge, 1) || !wide_fields(&big, 1)) return 1;
    if (!wide_fields(two, 2) || wide_fields(two, 1) || wide_fields(two, 0)) return 2;
    for (const ShotDesc &d : {narrow, odd})
        if (offset(d, 4 * d.nbx - 1, 4 * d.nby - 1, 4 * d.nbz - 1) != 64ll * d.nbx * d.nby * d.nbz - 1 ||
            64ll * d.nbz * d.nbx - 64 > 0x7fffffff) return 3;
    // the key of a captured iteration holds JacGeom's bytes
    JacGeom a{}, b{};
    b.wide = true;
    if (!std::memcmp(&a, &b, sizeof(a))) return 4;
    return 0;
}
"""


def test_offsets(tmp_path):
    (tmp_path / "o.cpp").write_text(SRC)
    exe = str(tmp_path / "o")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O0", "-I" + CSRC, "-I" + os.path.join(cuda, "include"), "-o", exe,
                    str(tmp_path / "o.cpp"), "-L" + os.path.join(cuda, "lib64"), "-lcudart"], check=True)
    assert subprocess.run([exe]).returncode == 0
    with open(os.path.join(CSRC, "api_iteration.cpp")) as f:
        assert "push(key_a, jg);" in f.read()
