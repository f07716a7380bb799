"""The reciprocal and quotient steps of the LU kernels (quotient.cuh) on the host: for every significand of the
divisor and every starting value within one unit in the last place of its reciprocal, the Newton step gives the
rounded reciprocal and the corrected quotient equals the division."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ops-blas_b200", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "quotient.cuh"
using namespace opsblas;
static float fl(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static uint32_t bits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
int main()
{
    long unusual = 0, starts = 0, reciprocals = 0, quotients = 0;
    uint64_t rng = 88172645463325252ull;
    for (uint32_t s = 0; s < (1u << 23); s++) {
        const float b = fl(0x3f800000u + s);  // 1 <= b < 2: a power of two scales every step exactly
        if (!qt_usual(b)) {
            unusual++;
            continue;
        }
        const float r = 1.0f / b;
        const double exact = 1.0 / (double)b, ulp = b == 1.0f ? 0x1p-23 : 0x1p-24;
        for (int d = -2; d <= 2; d++) {
            const float y0 = fl(bits(r) + d);
            if (fabs((double)y0 - exact) > ulp) continue;
            starts++;
            reciprocals += qt_newton(b, y0) != r;
        }
        for (int t = 0; t < 5; t++) {
            rng ^= rng << 13, rng ^= rng >> 7, rng ^= rng << 17;
            const uint32_t m = t == 0 ? 0u : t == 1 ? 0x7fffffu : t == 2 ? s : (uint32_t)(rng & 0x7fffffu);
            const float a = ldexpf(fl(0x3f800000u + m), -(int)((rng >> 30) % 60)) * ((rng >> 60) & 1 ? -1.0f : 1.0f);
            quotients += bits(qt_quotient(a, b, r)) != bits(a / b);
        }
    }
    // the ends of the range
    const bool ends = qt_usual(qt_low) && qt_usual(qt_high) && qt_usual(-qt_low) && !qt_usual(nextafterf(qt_low, 0.0f)) &&
                      !qt_usual(nextafterf(qt_high, INFINITY)) && !qt_usual(0.0f) && !qt_usual(NAN) && !qt_usual(INFINITY);
    printf("%ld %ld %ld %ld %d\n", unusual, starts, reciprocals, quotients, ends ? 1 : 0);
}
"""


def test_every_significand(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "q.cpp", tmp_path / "q"
    src.write_text(PROGRAM)
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-march=native", "-x", "c++", "-I", CSRC, str(src),
                           "-o", str(exe)])
    unusual, starts, reciprocals, quotients, ends = map(int, subprocess.check_output([str(exe)]).split())
    assert (reciprocals, quotients) == (0, 0)
    assert unusual == 1  # the significand of ones, which the theorem leaves out
    assert starts > 2 * (1 << 23) - 10
    assert ends == 1
