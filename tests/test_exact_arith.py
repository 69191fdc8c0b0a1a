"""The integer-pipe quotient and square root (swe_exact.cuh) on the CPU: compiled as plain C++ with the two
FP32 approximations off by up to two half units, bit for bit IEEE over random operands, equal and
all-ones or near-power-of-two significands, and operands whose result lies next to the midpoint of two
doubles (where the exact remainder decides)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "samoa_gb300", "csrc")

PROGRAM = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
namespace swe_exact {
typedef unsigned long long u64;
typedef long long s64;
static int off = 0;  // error added to the approximations, in units of 2^-24
static inline u64 bits_of(double x) { u64 r; memcpy(&r, &x, 8); return r; }
static inline double double_of(u64 v) { double r; memcpy(&r, &v, 8); return r; }
static inline float float_of(unsigned v) { float r; memcpy(&r, &v, 4); return r; }
static inline unsigned fbits_of(float x) { unsigned r; memcpy(&r, &x, 4); return r; }
static inline float ffma(float a, float b, float c) { return fmaf(a, b, c); }
static inline float fmul(float a, float b) { return a * b; }
static inline float fsub(float a, float b) { return a - b; }
static inline float ffromi(int v) { return (float)v; }
static inline float fclamp(float x, float lo, float hi) { return std::min(std::max(x, lo), hi); }
static inline float rcp32(float x) { return (float)(1.0 / x + off * 0x1p-24); }
static inline float rsqrt32(float x) { return (float)((1.0 + off * 0x1p-24) / sqrt((double)x)); }
static inline double ieee_div(double a, double b) { return a / b; }
static inline double ieee_sqrt(double x) { return sqrt(x); }
}
#include "swe_exact.cuh"
using namespace swe_exact;
static std::mt19937_64 g(11);
static u64 sig53(double x) { return (bits_of(x) & 0xfffffffffffffull) | (1ull << 52); }
static double draw() {
    u64 m = g() >> 12;
    switch (g() % 10) {
        case 0: m |= 0xffffffff00000ull; break;
        case 1: m &= 0xfffff00000000ull; break;
        case 2: m &= 0xf; break;
        case 3: m = 0xfffffffffffffull - (m & 0xf); break;
    }
    const int e = g() % 64 ? (int)(g() % 40) - 20 : (int)(g() % 2048) - 1023;  // subnormals, infinities, NaN too
    return double_of((u64)(e + 1023) << 52 | m | (g() & 1) << 63);
}
static double top53(unsigned __int128 p, int e) {
    while (p >> 53) p >>= 1;
    return ldexp((double)(u64)p, e);
}
static long bad = 0, fast = 0;
static void same(double got, double want) {
    if (bits_of(got) != bits_of(want) && !(std::isnan(got) && std::isnan(want)) && bad++ < 5) printf("%a want %a\n", got, want);
}
int main(int argc, char** argv) {
    off = atoi(argv[1]);
    for (long i = 0; i < atol(argv[2]); ++i) {
        const double b = draw();
        double a = draw(), x = fabs(draw());
        const u64 q = (g() >> 12) | (1ull << 52);
        if (i % 4 == 0) a = nextafter(top53((unsigned __int128)(2 * q + 1) * sig53(b), 5), g() & 1 ? INFINITY : 0);
        if (i % 4 == 1) x = top53((unsigned __int128)(2 * q + 1) * (2 * q + 1), (int)(g() % 9) - 52);
        if (i % 4 == 1 && (g() & 1)) x = nextafter(x, INFINITY);
        if (i % 16 == 2) a = ldexp(b, 3);
        if (i % 64 == 3) a = 0.0 * a;
        const u64 y = recip_fix(b);
        same(div_fix(a, b, y), a / b);
        same(sqrt_fix(x), sqrt(x));
        same(sqrt_fix(a), sqrt(a));
        FastOps f;
        const double fq = f.div(a, recip_of(b)), f1 = f.div1(b, x), fr = f.sqrt(x);
        if (f.ok) same(fq, a / b), same(f1, b / x), same(fr, sqrt(x)), ++fast;
        if (y && llabs((long long)(bits_of(recip_near(b, y)) - bits_of(1.0 / b))) > 1) ++bad;
    }
    printf("%ld differ, %ld fast\n", bad, fast);
    return bad != 0 || fast < atol(argv[2]) / 2;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact")
    (d / "check.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", str(d / "check"),
                           str(d / "check.cpp")])
    return str(d / "check")


@pytest.mark.parametrize("off", [-2, 0, 2])
def test_quotient_and_root_are_ieee(program, off):
    r = subprocess.run([program, str(off), "1500000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
