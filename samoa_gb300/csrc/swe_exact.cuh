// Correctly rounded FP64 quotients and square roots on the integer and FP32
// pipes.
//
// GB300 retires one FP64 warp instruction per SM in 16 cycles (measured: 501e9
// FP64 lane-instructions/s) against 4 integer or FP32 warp instructions per
// cycle, so one FP64 instruction costs as much issue time as 64 others. An IEEE
// quotient from a shared reciprocal takes 5 FP64 instructions (6 more for the
// reciprocal), an IEEE square root about 8. Here both take none: the
// significands are integers, an approximation to about 62 bits comes from the
// FP32 reciprocal (or reciprocal square root) and one or two Newton steps whose
// residuals are formed exactly modulo 2^64. Its top 53 bits or their successor
// are the result, and the sign of the exact remainder against the midpoint
// between the two says which (the usual remainder test of a rounding, as in
// Muller et al., Handbook of Floating-Point Arithmetic, on "division" and
// "square root"; neither a quotient nor a square root of 53-bit significands is
// ever a midpoint itself). So every result is RN(a / b) or RN(sqrt(x)), bit for
// bit; operands outside the handled range take the IEEE operation.
//
// The cores have no branches: a branch ends a basic block, and with one in every
// quotient and root the compiler could not overlap their chains (a chain of about
// 100 to 150 cycles each) with each other or with the FP64 instructions, of
// which a warp can start one per 64 cycles. FastOps therefore only notes that an
// operand was out of range, and the caller redoes such an edge with SafeOps.
//
// Plain C++ apart from the few shims below, so that the CPU can check it with
// worst-case errors of the two FP32 approximations.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define SWE_EXACT_FN __device__ __forceinline__
#define SWE_EXACT_FN_M __device__ __forceinline__
#else
#define SWE_EXACT_FN static inline
#define SWE_EXACT_FN_M inline
#endif

namespace swe_exact {

typedef unsigned long long u64;
typedef long long s64;

#ifdef __CUDACC__
// Casts the compiler cannot see through: a test on the bits stays an integer
// instruction (with the plain casts it may come back as an FP64 comparison).
SWE_EXACT_FN u64 bits_of(double x) {
    u64 r;
    asm("mov.b64 %0, %1;" : "=l"(r) : "d"(x));
    return r;
}
SWE_EXACT_FN double double_of(u64 v) {
    double r;
    asm("mov.b64 %0, %1;" : "=d"(r) : "l"(v));
    return r;
}
SWE_EXACT_FN float float_of(unsigned v) { return __uint_as_float(v); }
SWE_EXACT_FN unsigned fbits_of(float x) { return __float_as_uint(x); }
SWE_EXACT_FN float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
SWE_EXACT_FN float fmul(float a, float b) { return __fmul_rn(a, b); }
SWE_EXACT_FN float fsub(float a, float b) { return __fsub_rn(a, b); }
SWE_EXACT_FN float ffromi(int v) { return __int2float_rn(v); }
SWE_EXACT_FN float fclamp(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }
SWE_EXACT_FN float rcp32(float x) {  // within 2^-23 on [1, 2]
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
SWE_EXACT_FN float rsqrt32(float x) {  // within 2^-22.9 relative
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
SWE_EXACT_FN double ieee_div(double a, double b) { return a / b; }
SWE_EXACT_FN double ieee_sqrt(double x) { return sqrt(x); }
#endif

// 12582912 = 1.5 * 2^23: adding it to |x| < 2^22 leaves RN(x) in the low bits.
constexpr float kMagic = 12582912.0f;
constexpr unsigned kMagicBits = 0x4b400000u;

// 2^64 / m, m in [1, 2) the significand of b, with an error in (-2, 1) (2^64 - 1
// for m = 1); 0 for a b whose exponent is outside [-500, 500] (zero, subnormal,
// infinite and NaN among them), which says: take the IEEE division.
SWE_EXACT_FN u64 recip_fix(double b) {
    const u64 ub = bits_of(b);
    const unsigned hi = (unsigned)(ub >> 32), lo = (unsigned)ub;
    const unsigned e = (hi >> 20) & 0x7ffu;
    // m = fb + fl 2^-23 (+ less than 2^-46)
    const float fb = float_of(0x3f800000u | (((hi << 3) | (lo >> 29)) & 0x7fffffu));
    const float fl = fsub(float_of(0x3f800000u | ((lo & 0x1fffffffu) >> 6)), 1.0f);
    const float y0 = fclamp(rcp32(fb), 0.5f, 1.0f);  // within 2^-22 of 1 / m, a multiple of 2^-24
    float r = ffma(-fb, y0, 1.0f);
    r = ffma(fmul(fl, -1.1920928955078125e-07f), y0, r);  // 1 - m y0 to about 2^-45
    // y1 = y0 + y0 r as an integer multiple of 2^-43 (|y0 r| 2^43 < 2^22), within 2^-42 of 1 / m
    const int n = (int)(fbits_of(ffma(y0, fmul(r, 8796093022208.0f), kMagic)) - kMagicBits);
    const u64 y1 = ((u64)(fbits_of(y0) - 0x3e800000u) << 19) + (u64)(s64)n;
    // 2^95 (1 - m y1), below 2^54 in magnitude, exact modulo 2^64
    const u64 mb = (ub & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const s64 d = (s64)(0ull - mb * y1);
    const s64 c = (s64)(int)(d >> 24) * (s64)(int)(y1 >> 13);
    u64 y = (y1 << 21) + (u64)(c >> 37);
    if ((ub & 0x000fffffffffffffull) == 0) y = ~0ull;
    return e - 523u <= 1000u ? y : 0ull;
}

// RN(a / b) for normal a and b of exponents within [-500, 500], y = recip_fix(b).
SWE_EXACT_FN double quot_core(u64 ua, u64 ub, u64 y) {
    // the quotient of the significands times 2^63, low by less than 5 or high by less
    // than 1 (the lowest partial product is left out), then normalised to [2^63, 2^64)
    const unsigned ah = (unsigned)(ua >> 21) | 0x80000000u, al = (unsigned)ua << 11;
    const unsigned yh = (unsigned)(y >> 32), yl = (unsigned)y;
    u64 q = (u64)ah * yh + (((u64)ah * yl >> 32) + ((u64)al * yh >> 32));
    const unsigned s = (unsigned)(q >> 63);
    q <<= 1u - s;
    // r or r + 1, r = q >> 11: by the sign of a 2^(54 - s) - b (2 r + 1), below 2^54 in
    // magnitude, from its bits modulo 2^64
    const u64 mb = (ub & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const u64 p = mb * ((q >> 10) | 1u);
    const unsigned up = ((unsigned)(p >> 32) - ((unsigned)ua << (22u - s))) >> 31;
    const unsigned e = ((unsigned)(ua >> 52) & 0x7ffu) - ((unsigned)(ub >> 52) & 0x7ffu) + 1021u + s;
    return double_of((((u64)e << 52) + ((q >> 11) + up)) | ((ua ^ ub) & 0x8000000000000000ull));
}

// RN(a / b) from y = recip_fix(b).
SWE_EXACT_FN double div_fix(double a, double b, u64 y) {
    const u64 ua = bits_of(a), ub = bits_of(b);
    const unsigned ea = (unsigned)(ua >> 52) & 0x7ffu, eb = (unsigned)(ub >> 52) & 0x7ffu;
    if (ea - 523u > 1000u || y == 0) {
        if ((ua << 1) == 0 && eb - 1u < 2046u) return double_of((ua ^ ub) & 0x8000000000000000ull);  // +-0 / b
        return ieee_div(a, b);
    }
    return quot_core(ua, ub, y);
}

// RN(a / b) for a divisor of its own.
SWE_EXACT_FN double div_one(double a, double b) { return div_fix(a, b, recip_fix(b)); }

// The double nearest (to within 0.51 ulp) to 1 / b from y = recip_fix(b), for
// values that need no correct rounding.
SWE_EXACT_FN double recip_near(double b, u64 y) {
    if (y == 0) return ieee_div(1.0, b);
    const u64 ub = bits_of(b);
    const unsigned eb = (unsigned)(ub >> 52) & 0x7ffu;
    const u64 r = (y >> 11) + ((y >> 10) & 1u);  // 2^53 / m, in (2^52, 2^53]
    return double_of((((u64)(2044u - eb) << 52) + r) | (ub & 0x8000000000000000ull));
}

// RN(sqrt(x)) for a positive normal x.
SWE_EXACT_FN double root_core(u64 ux) {
    const unsigned hi = (unsigned)(ux >> 32), lo = (unsigned)ux;
    const unsigned e = hi >> 20;
    // x = M 4^k with M in [1, 4): M 2^52 is m
    const unsigned odd = (e & 1u) ^ 1u;
    const u64 m = ((ux & 0x000fffffffffffffull) | 0x0010000000000000ull) << odd;
    const float fm = float_of((0x3f800000u + (odd << 23)) | (((hi << 3) | (lo >> 29)) & 0x7fffffu));
    const float r0 = fclamp(rsqrt32(fm), 0.5f, 1.0f);  // 1 / sqrt(M) to 2^-22 relative, a multiple of 2^-24
    const float f1 = fclamp(fmul(fm, r0), 1.0f, 2.0f);
    const unsigned s1 = fbits_of(f1) - 0x3f000000u;    // sqrt(M) 2^23, within 2^-21
    // Heron with 1 / s = r0: the residual M - s1^2 is exact, |d1| < 2^33 at scale 2^52
    const s64 d1 = (s64)(m - ((u64)s1 * s1 << 6));
    // s2 = s1 + d1 r0 / 2 as a multiple of 2^-42 (d1 r0 2^-11 < 2^22), within 2^-42
    const float t = fmul(ffromi((int)(d1 >> 3)), r0);
    const int n = (int)(fbits_of(ffma(t, 0.00390625f, kMagic)) - kMagicBits);
    const u64 s2 = ((u64)s1 << 19) + (u64)(s64)n;
    // again: |d2| < 2^45 at scale 2^84, exact modulo 2^64; s = s2 + d2 r0 / 2 at scale 2^63
    const s64 d2 = (s64)((m << 32) - s2 * s2);
    const s64 c = (s64)(int)(d2 >> 14) * (s64)(int)(fbits_of(r0) - 0x3e800000u);
    const u64 s = (s2 << 21) + (u64)(c >> 32);  // error within 3
    // r or r + 1, r = s >> 11: by the sign of M 2^106 - (2 r + 1)^2
    const u64 h = (s >> 10) | 1u, p = h * h;
    const unsigned up = ((unsigned)(p >> 32) - ((unsigned)m << 22)) >> 31;
    return double_of(((u64)((e + 1021u - odd) >> 1) << 52) + ((s >> 11) + up));
}

// RN(sqrt(x)).
SWE_EXACT_FN double sqrt_fix(double x) {
    const u64 ux = bits_of(x);
    // with the sign bit: negative x fails the range test
    if ((unsigned)(ux >> 52) - 1u >= 2046u) return (ux << 1) == 0 ? x : ieee_sqrt(x);
    return root_core(ux);
}

// A divisor with its reciprocal (recip_fix; 0 where it was left out or is out of range).
struct Recip {
    double b;
    u64 y;
};
SWE_EXACT_FN Recip recip_of(double b) { return Recip{b, recip_fix(b)}; }

// The quotients and roots of a formula, for every operand.
struct SafeOps {
    static constexpr bool kFast = false;
    bool ok = true;
    SWE_EXACT_FN_M double div(double a, const Recip& r) { return div_fix(a, r.b, r.y); }
    SWE_EXACT_FN_M double div1(double a, double b) { return div_one(a, b); }
    // a / b where `use`, else any value; div_if: b a depth above a tolerance >= 0
    SWE_EXACT_FN_M double div_if(bool use, double a, const Recip& r) { return use ? div_fix(a, r.b, r.y) : 0.0; }
    SWE_EXACT_FN_M double div1_if(bool use, double a, double b) { return use ? div_one(a, b) : 0.0; }
    SWE_EXACT_FN_M double sqrt(double x) { return sqrt_fix(x); }
};

// The same without branches (and without the short-circuit tests that may become some);
// ok is false after an operand that SafeOps has to take.
struct FastOps {
    static constexpr bool kFast = true;
    bool ok = true;
    SWE_EXACT_FN_M double quot(bool use, bool zero_free, double a, const Recip& r) {
        const u64 ua = bits_of(a), ub = bits_of(r.b);
        const bool zero = (ua << 1) == 0;
        const bool in = ((unsigned)(ua >> 52) & 0x7ffu) - 523u <= 1000u;
        const bool y = r.y != 0;
        ok = ok & (!use | (zero ? (zero_free | y) : (in & y)));
        const double q = quot_core(ua, ub, r.y);
        return zero ? double_of((ua ^ ub) & 0x8000000000000000ull) : q;
    }
    SWE_EXACT_FN_M double div(double a, const Recip& r) { return quot(true, false, a, r); }
    SWE_EXACT_FN_M double div1(double a, double b) { return quot(true, false, a, recip_of(b)); }
    SWE_EXACT_FN_M double div_if(bool use, double a, const Recip& r) { return quot(use, true, a, r); }
    SWE_EXACT_FN_M double div1_if(bool use, double a, double b) { return quot(use, false, a, recip_of(b)); }
    SWE_EXACT_FN_M double sqrt(double x) {
        const u64 ux = bits_of(x);
        ok = ok & ((unsigned)(ux >> 52) - 1u < 2046u);
        return root_core(ux);
    }
};

}  // namespace swe_exact
