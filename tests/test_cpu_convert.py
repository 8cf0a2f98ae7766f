"""The kernels' integer conversions between FP64 and FP32 give the casts' results bit for bit (any
NaN for a NaN), compiled for the host: random bit patterns, every exponent of the FP32 range with
halves and sparse low parts (differences of two positions, as the positions' hi/lo split forms
them), denormals, overflow, infinities; FP32 to FP64 over a grid through all patterns."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "md_tian2_gb300" / "csrc"

SOURCE = r"""
#include "mdt_convert.h"
#include <cmath>
#include <cstdio>
#include <random>
using namespace mdt;
static long bad = 0;
static void narrow(double x) {
    const float a = f32_of(x), b = (float)x;
    if (std::isnan(b) ? !std::isnan(a) : bits_of(a) != bits_of(b)) bad += 1;
}
static void widen(float x) {
    const double a = f64_of(x), b = (double)x;
    if (std::isnan(b) ? !std::isnan(a) : bits_of(a) != bits_of(b)) bad += 1;
}
static void split(double x, double y, double z) {
    float h[3], l[3];
    split3(x, y, z, h, l);
    const double p[3] = {x, y, z};
    for (int d = 0; d < 3; ++d) {
        const float a = (float)p[d], b = (float)(p[d] - (double)a);
        bad += std::isnan(a) ? !std::isnan(h[d]) : bits_of(a) != bits_of(h[d]);
        bad += std::isnan(b) ? !std::isnan(l[d]) : bits_of(b) != bits_of(l[d]);
    }
}
int main() {
    std::mt19937_64 g(1);
    for (int i = 0; i < 1000000; ++i) {
        uint64_t u = g();
        double x;
        std::memcpy(&x, &u, 8);
        narrow(x);
        const uint64_t e = 0x360 + g() % 0x130;  // 2^-159 .. 2^144
        uint64_t f = g() & 0xfffffffffffffull;
        if (i & 1) f = (f & ~0x1fffffffull) | 0x10000000ull;
        u = (g() & 1) << 63 | e << 52 | f;
        std::memcpy(&x, &u, 8);
        narrow(x);
        const double r = std::ldexp((double)(g() >> 11), -49);  // a position, its high part, the rest
        narrow(r - f64_of(f32_of(r)));
        split(x, r, -r);
    }
    for (uint64_t u = 0; u < 1ull << 32; u += 997) widen(float_of_bits((uint32_t)u));
    for (uint32_t u : {0u, 1u, 0x007fffffu, 0x00800000u, 0x7f7fffffu, 0x7f800000u, 0x7f800001u, 0x7fc00000u})
        for (uint32_t s : {0u, 0x80000000u}) {
            const float f = float_of_bits(u | s);
            widen(f);
            narrow((double)f);
            for (double w : {0.5, 0.75, 1.5}) narrow((double)f * w);
        }
    for (double x : {0.0, -0.0, 0x1p-150, 0x1.8p-150, 0x1p-149, -0x1.8p-149, 0x1.fffffffp-127, 0x1.ffffffp127, 0x1.fffffefffffffp127, 0x1p128, 0x1p-1074})
        narrow(x), narrow(-x), split(x, 1.0, -x), split(0.1, x, 3e-23);
    std::printf("%ld\n", bad);
    return 0;
}
"""


def test_integer_conversions(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    (tmp_path / "convert.cpp").write_text(SOURCE)
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", str(CSRC), str(tmp_path / "convert.cpp"), "-o", str(tmp_path / "convert")],
                   check=True)
    out = subprocess.run([str(tmp_path / "convert")], check=True, capture_output=True, text=True)
    assert int(out.stdout) == 0
