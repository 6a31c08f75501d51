"""The three-operation division of csrc/common.cuh (q = RN(a z), r = a - q y, RN(q + r z) with
z = RN(1 / y)) against the IEEE quotient, restated in C with fmaf.

q + r z differs from a / y by less than 3 x 2^-25 ulp, so the only quotients that could round
the other way lie that near a midpoint of two floats.  `midpoints` solves for them: for every
24-bit divisor Y and every small k, the X with X 2^s - M Y = k, M odd -- all cases with |k| up
to 11 where |k| <= 2 is needed -- and compares each.  `all_dividends` goes through every
mantissa of the dividend for spacings in use and some others.
"""
import ctypes
import subprocess

import pytest

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
static float bits(unsigned u) { float x; memcpy(&x, &u, 4); return x; }
static float three(float a, float y, float z) { float q = a * z, r = fmaf(-q, y, a); return fmaf(r, z, q); }
long midpoints(long *bad, int s)  /* s = 25: X < Y, quotients in [1/2, 1); s = 24: in [1, 2) */
{
    long seen = 0;
    *bad = 0;
    for (uint64_t Y = 1u << 23; Y < (1u << 24); Y++) {
        const float y = ldexpf((float)Y, -23), z = 1.0f / y;
        const int t = __builtin_ctzll(Y);
        for (int64_t k = -11; k <= 11; k++) {
            if (!k || k % (1ll << t)) continue;
            const uint64_t mod = (1ull << s) >> t, Yo = Y >> t;
            uint64_t inv = Yo;
            for (int i = 0; i < 5; i++) inv *= 2 - Yo * inv;
            for (uint64_t M = ((uint64_t)(-(k >> t)) * inv) & (mod - 1); M < (1ull << 25); M += mod) {
                const uint64_t v = M * Y + (uint64_t)k, X = v >> s;
                if (M < (1ull << 24) || !(M & 1) || (v & ((1ull << s) - 1)) || X < (1u << 23) || X >= (1u << 24)) continue;
                if ((s == 25) != (X < Y)) continue;
                const float x = ldexpf((float)X, -23);
                seen++;
                if (three(x, y, z) != x / y) ++*bad;
            }
        }
    }
    return seen;
}
long all_dividends(float y)
{
    const float z = 1.0f / y;
    long bad = 0;
    for (unsigned m = 0; m < (1u << 23); m++) {
        const float a = bits(0x3f800000u | m), b = bits(0x17800000u | m);
        bad += three(a, y, z) != a / y;
        bad += three(b, y, z) != b / y;
        bad += three(-b, y, z) != -b / y;
    }
    return bad + (three(0.0f, y, z) != 0.0f);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("divide")
    (d / "d.c").write_text(SRC)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(d / "d.so"), str(d / "d.c"), "-lm"]
                   + (["-mfma"] if "fma" in open("/proc/cpuinfo").read() else []), check=True)
    so = ctypes.CDLL(str(d / "d.so"))
    so.midpoints.restype = so.all_dividends.restype = ctypes.c_long
    so.midpoints.argtypes = [ctypes.POINTER(ctypes.c_long), ctypes.c_int]
    so.all_dividends.argtypes = [ctypes.c_float]
    return so


@pytest.mark.parametrize("shift", [24, 25])
def test_quotients_near_a_midpoint(lib, shift):
    bad = ctypes.c_long()
    assert lib.midpoints(ctypes.byref(bad), shift) > 1_000_000
    assert bad.value == 0


@pytest.mark.parametrize("y", [10.0, 12.5, 20.0, 25.0, 50.0, 51.0, 52.0, 7.3, 0.1, 1.0, 1.9999999, 1.0000001, 333.33,
                               2.0 ** -40, 2.0 ** 40])
def test_every_dividend(lib, y):
    assert lib.all_dividends(y) == 0
