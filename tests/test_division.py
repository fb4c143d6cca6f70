"""div_small and div_rn (csrc/mpp_div.cuh) against the IEEE division, compiled for the CPU: every mantissa for
every small divisor, signs, zeros, subnormals and random operands over the stated ranges are the same bit for bit
(but the sign of a zero); what is infinite or NaN stays one of the two."""
import os
import subprocess

from conftest import PKG

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#define __device__
#define __forceinline__ inline
#include "mpp_div.cuh"
static float f(uint32_t b) { float x; memcpy(&x, &b, 4); return x; }
static uint32_t bits(float x) { uint32_t b; memcpy(&b, &x, 4); return b; }
static long bad = 0;
static void check(const char* what, float got, float a, float d, long ulps = 0) {
    const float want = a / d;
    if (got == want || (!std::isfinite(got) && !std::isfinite(want))) return;
    if (std::isfinite(got) && std::isfinite(want) && labs((long)bits(got) - (long)bits(want)) <= ulps) return;
    if (bad++ < 20) printf("%s %a / %a: %a, not %a\n", what, a, d, got, want);
}
int main() {
    const float special[] = {INFINITY, -INFINITY, NAN, 0.f, -0.f, 3.4028234e38f, -3.4028234e38f, 1.1754944e-38f};
    std::mt19937 g(1);
    for (int n = 1; n <= 6; n++) {
        const float d = (float)n, rd = 1.f / d;
        for (uint32_t m = 0; m < (1u << 23); m++) check("small", mpp::div_small(f(0x3f800000u | m), d, rd), f(0x3f800000u | m), d);
        for (float a : special) check("small", mpp::div_small(a, d, rd), a, d);
        for (uint32_t m = 0; m < (1u << 24); m += 7)  // quotients below 2^-126: ties of d = 6 may go the other way
            check("small", mpp::div_small(f(m), d, rd), f(m), d, n == 6 ? 1 : 0);
        for (int i = 0; i < 1000000; i++) {
            const float a = f((uint32_t)g());
            check("small", mpp::div_small(a, d, rd), a, d, n == 6 && std::fabs(a) < 0x1p-123f ? 1 : 0);
        }
    }
    std::uniform_int_distribution<uint32_t> de(127 - 30, 127 + 29), ae(127 - 70, 254);
    for (int i = 0; i < 6000000; i++) {
        float d = f(de(g) << 23 | ((uint32_t)g() & 0x7fffffu));
        if (i % 16 == 0) d = f(bits(d) | 0x7fffffu);
        float a = f(ae(g) << 23 | ((uint32_t)g() & 0x807fffffu));
        if (i % 64 == 0) a = special[i / 64 % 7];
        check("any", mpp::div_rn(a, d, 1.f / d), a, d);
    }
    return bad ? 1 : 0;
}
"""


def test_division_rounds_as_ieee(tmp_path):
    src, exe = tmp_path / "division.cpp", tmp_path / "division"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(PKG, "csrc"), "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
