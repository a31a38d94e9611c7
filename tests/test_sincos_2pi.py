"""The normal transform's sine and cosine, compiled for the host (every operation is a correctly rounded
float one): within 1.5 ulp of the 64-bit functions of the rounded angle, on every float u next to
1/4, 1/2 and 3/4, where one of them is as small as 1e-8, and on a sample of all others."""
from __future__ import annotations

import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "remora_b200" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#define __device__
#define __forceinline__ inline
static int __float_as_int(float f) { int i; std::memcpy(&i, &f, 4); return i; }
static float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }
static float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
#include "sincos_2pi.cuh"
static double ulps(float got, long double want) {
    const float w = std::fabs((float)want);
    return std::fabs((double)((long double)got - want)) / ((double)std::nextafter(w, INFINITY) - w);
}
int main() {
    double near = 0, all = 0;
    auto look = [](double& worst, float u) {
        float s, c;
        rc::sincos_2pi(u, &s, &c);
        const long double q = (2.0f * 3.14159265358979323846f) * u;
        worst = std::fmax(worst, std::fmax(ulps(s, std::sin(q)), ulps(c, std::cos(q))));
    };
    for (float at : {0.25f, 0.5f, 0.75f})
        for (int d = -20000; d <= 20000; ++d) look(near, __int_as_float(__float_as_int(at) + d));
    for (int b = __float_as_int(0x1p-6f); b < __float_as_int(1.0f); b += 61) look(all, __int_as_float(b));
    for (int b = __float_as_int(0x1p-32f); b < __float_as_int(0x1p-6f); b += 257) look(all, __int_as_float(b));
    std::printf("%.4f %.4f", near, all);
}
"""


def test_within_one_and_a_half_ulp(tmp_path):
    src, exe = tmp_path / "a.cpp", tmp_path / "a.out"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    near, everywhere = map(float, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert near <= 1.5 and everywhere <= 1.5, (near, everywhere)
