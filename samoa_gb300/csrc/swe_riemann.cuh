// Device-side edge fluxes of the SWE step: the GeoClaw double-precision Riemann
// solvers and the Lax-Friedrichs fluxes, evaluated per edge in FP64.
//
// Bit-for-bit agreement with the CPU restatement needs the same rounding at
// every operation: this file is compiled with --fmad=false (no contraction)
// and keeps the reference's left-to-right evaluation order of each expression.
// Sums written in the reference as dot_product/matmul start from +0.0; that
// first addition only turns a -0.0 into +0.0, which z0() does with integer
// instructions instead of spending an FP64 add.
#pragma once

// The kernels are compiled twice: in namespace swe with strict IEEE rounding
// (no contraction) and in namespace swe_fma with FMA contraction (SWE_KNS).
#ifndef SWE_KNS
#define SWE_KNS swe
#endif
namespace swe {}

#include <stdint.h>

#include "swe_exact.cuh"

namespace SWE_KNS {
using namespace ::swe;
using namespace ::swe_exact;

constexpr double kG = 9.80665;  // src/SWE/SWE_data_types.f90:34

enum Solver : int { FWAVE = 1, AUG_RIEMANN = 3, LF = 10, LF_BATH = 11, LLF = 12, LLF_BATH = 13 };
enum Boundary : int { BC_OUTFLOW = 0, BC_SLIP = 1, BC_NOSLIP = 2 };

struct State {
    double h, p1, p2, b;  // surface elevation (or the depth: edge_flux's SURFACE), momentum, bathymetry
};
struct Update {
    double h, p1, p2, s;  // net update (or flux) and maximum wave speed
};

// Bit casts the compiler cannot see through: tests on the bit pattern of a double
// stay integer instructions (with the plain casts the compiler may turn a test
// such as "bits << 1 == 0" back into an FP64 comparison, on the FP64 pipe).
__device__ __forceinline__ long long dbits(double x) {
    long long r;
    asm("mov.b64 %0, %1;" : "=l"(r) : "d"(x));
    return r;
}
__device__ __forceinline__ double bitsd(long long v) {
    double r;
    asm("mov.b64 %0, %1;" : "=d"(r) : "l"(v));
    return r;
}

__device__ __forceinline__ double z0(double x) {
    long long v = dbits(x);
    return bitsd(v == (long long)0x8000000000000000ULL ? 0LL : v);
}
// The step's products, named by where they are taken (the solver's, the edge
// rotations', the cell update's): plain FP64 multiplies. Moving them to the
// integer pipe was measured slower (see the design notes of the FP64 diet).
__device__ __forceinline__ double prod(double a, double b) { return a * b; }
__device__ __forceinline__ double prod_rot(double a, double b) { return a * b; }
__device__ __forceinline__ double prod_cell(double a, double b) { return a * b; }

__device__ __forceinline__ double dmn(double a, double b) { return (a < b) ? a : b; }
__device__ __forceinline__ double dmx(double a, double b) { return (a > b) ? a : b; }

// IEEE predicates on the integer pipe (bit patterns), exact for every input
// including +-0, infinities and NaN; the FP64 pipe is the step's bottleneck.
__device__ __forceinline__ long long abs_bits(double x) { return dbits(x) & 0x7fffffffffffffffLL; }
__device__ __forceinline__ bool not_nan(long long a) { return a <= 0x7ff0000000000000LL; }  // a = abs_bits
__device__ __forceinline__ bool is_finite(double x) { return abs_bits(x) < 0x7ff0000000000000LL; }
__device__ __forceinline__ bool lt0(double x) {  // x < 0.0
    const long long b = dbits(x);
    const long long a = b & 0x7fffffffffffffffLL;
    return (b < 0) & (a != 0) & not_nan(a);
}
__device__ __forceinline__ bool gt0(double x) {  // x > 0.0
    const long long b = dbits(x);
    return (b > 0) & (b <= 0x7ff0000000000000LL);
}
__device__ __forceinline__ bool is_nan(double x) { return abs_bits(x) > 0x7ff0000000000000LL; }
// A key that orders like the value for non-NaN doubles, with -0 equal to +0.
__device__ __forceinline__ long long ord_key(double x) {
    long long b = dbits(x);
    b = (b == (long long)0x8000000000000000ULL) ? 0LL : b;
    return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}
__device__ __forceinline__ bool lt(double a, double b) {  // a < b
    return !is_nan(a) & !is_nan(b) & (ord_key(a) < ord_key(b));
}
__device__ __forceinline__ double imin(double a, double b) { return lt(a, b) ? a : b; }  // dmn on the integer pipe
__device__ __forceinline__ double imax(double a, double b) { return lt(b, a) ? a : b; }  // dmx on the integer pipe
// x with its sign flipped when `neg` (exact, like multiplying by -1)
__device__ __forceinline__ double flip(double x, bool neg) {
    return bitsd(dbits(x) ^ (neg ? (long long)0x8000000000000000ULL : 0LL));
}
// `SWE_IF(c) { ... }` is `if (c) { ... }` that stays a branch: a loop whose end the
// compiler cannot see. Conditional FP64 code needs it. The compiler turns short
// conditional blocks into predicated instructions, and a predicated FP64
// instruction holds the FP64 pipe for its 16 to 19 cycles per warp and SM even
// when no lane executes it (measured: one or six multiplies behind an `if`, a warp
// vote or a bra.uni that is never taken cost as much as multiplies always done).
__device__ __forceinline__ unsigned int opaque_zero() {
    unsigned int v;
    asm volatile("mov.u32 %0, 0;" : "=r"(v));
    return v;
}
#define SWE_IF(c) for (unsigned int swe_if_ = (c) ? 1u : 0u; swe_if_; swe_if_ = opaque_zero())

// x + z for z = +-0, as IEEE addition gives it: x itself, except that a zero x
// takes +0 unless both are -0, and a NaN x comes back quiet.
__device__ __forceinline__ double add_zero(double x, double z) {
    const long long b = dbits(x);
    if ((b << 1) == 0) return bitsd(b & dbits(z));  // -0 only when both are -0
    return abs_bits(x) > 0x7ff0000000000000LL ? bitsd(b | 0x0008000000000000LL) : x;
}
// RN(x * p) for p = 2^k: while x and the result are normal numbers the product
// is exact and only the exponent field moves (an integer add on the bit
// pattern); +-0 stays itself; a subnormal, infinite or NaN operand and an
// under- or overflowing result take the FP64 multiply.
__device__ __forceinline__ bool scales(long long b, int k) {  // a zero, or normal before and after
    const int e = (int)((b >> 52) & 0x7ff);
    return ((b << 1) == 0) | (((unsigned)(e - 1) <= 2045u) & ((unsigned)(e + k - 1) <= 2045u));
}
__device__ __forceinline__ double scaled(long long b, int k) {
    return bitsd((b << 1) == 0 ? b : b + ((long long)k << 52));
}
__device__ __forceinline__ double scale_pow2(double x, int k, double p) {
    double r = scaled(dbits(x), k);
    SWE_IF(!scales(dbits(x), k)) r = x * p;
    return r;
}

// Several quotients in the step share a divisor (a cell's depth divides its
// edges' normal and tangential momenta; the two f-wave coefficients share
// s2 - s1): a Recip is the divisor with its reciprocal (swe_exact.cuh).
__device__ __forceinline__ double div_rn(double a, const Recip& r) { return div_fix(a, r.b, r.y); }
// 1 / b to about half an ulp, for cotangents, which need no correct rounding
__device__ __forceinline__ double rcp_near(double b) { return recip_near(b, recip_fix(b)); }

// Non-strict comparisons on the integer pipe with IEEE semantics (false if either is NaN).
__device__ __forceinline__ bool le(double a, double b) {  // a <= b
    return !is_nan(a) & !is_nan(b) & (ord_key(a) <= ord_key(b));
}
// The predicates on numbers, for FastOps formulas: a NaN operand gives any answer
// there, and the formula is then redone (FastOps::ok is false: every value
// compared reaches a divisor, a dividend or a root, and none of those takes a NaN).
__device__ __forceinline__ long long num_key(double x) {
    const long long b = dbits(x), m = b & 0x7fffffffffffffffLL, t = b >> 63;
    return (m ^ t) - t;
}
template <class Ops>
__device__ __forceinline__ bool olt(double a, double b) { return Ops::kFast ? num_key(a) < num_key(b) : lt(a, b); }
template <class Ops>
__device__ __forceinline__ bool ole(double a, double b) { return Ops::kFast ? num_key(a) <= num_key(b) : le(a, b); }
template <class Ops>
__device__ __forceinline__ bool olt0(double x) {
    return Ops::kFast ? (dbits(x) < 0) & ((dbits(x) << 1) != 0) : lt0(x);
}
template <class Ops>
__device__ __forceinline__ bool ogt0(double x) { return Ops::kFast ? dbits(x) > 0 : gt0(x); }
// RN(x 2^k), p = 2^k
template <class Ops>
__device__ __forceinline__ double oscale(double x, int k, double p, Ops& o) {
    if (!Ops::kFast) return scale_pow2(x, k, p);
    o.ok = o.ok & scales(dbits(x), k);
    return scaled(dbits(x), k);
}
template <class Ops>
__device__ __forceinline__ double omin(double a, double b) { return olt<Ops>(a, b) ? a : b; }
template <class Ops>
__device__ __forceinline__ double omax(double a, double b) { return olt<Ops>(b, a) ? a : b; }
__device__ __forceinline__ double iabs(double x) { return bitsd(abs_bits(x)); }  // fabs

// The branch decisions of one augmented-solver evaluation, for its reverse
// (the discrete adjoint re-evaluates the values; the decisions fix the branch).
struct AugRec {
    int8_t rs;        // riemanntype: 0 a side at most dry, 1 two rarefactions, 2 two shocks, 3 one of each
    bool lowR, highR;  // h_min resp. h_max is hR
    bool lhigh;        // one of each: hL > hR
    bool t_pos;        // two rarefactions: t = -delu + 2 (sqL + sqR) kept (not the 0)
    bool l0_sE1, l2_sE2, hst_pos, hbar_pos, tilde_x, sonic;
    int8_t dcase;      // deldelh bounds: 0 none, 1 both speeds apart, 2 sE1 >= ct, 3 sE2 <= -ct
    bool dd_min_first, dd_max_first;  // each bound kept the running value
    bool ph_mx_pl, ph_min_first, ph_mn_pl, ph_max_first;  // deldelphi bounds
    double s1m, s2m;   // riemanntype's speeds
};

// Riemann structure with one Newton step, src/geoclaw/riemannsolvers.f:507-618.
// sqL / sqR are sqrt(g * hL) and sqrt(g * hR) (the caller's, the same operands
// and so the same bits as computing them here); yL / yR are recip_fix of hL / hR
// (0: the IEEE division).
template <bool REC, class Ops>
__device__ __forceinline__ void riemann_structure_rec(double hL, double hR, double uL, double uR, double drytol,
                                                     double sqL, double sqR, u64 yL, u64 yR, double& hm, double& s1m, double& s2m,
                                                     AugRec* rec, Ops& o) {
    const double g = kG;
    const bool r_lower = olt<Ops>(hR, hL);  // h_min = dmn(hR, hL) is hR
    const double h_min = r_lower ? hR : hL, sq_min = r_lower ? sqR : sqL;
    const bool r_higher = olt<Ops>(hL, hR);  // h_max = dmx(hR, hL) is hR
    const double h_max = r_higher ? hR : hL, sq_max = r_higher ? sqR : sqL;
    if (REC) {
        rec->lowR = r_lower;
        rec->highR = r_higher;
    }
    double delu = uR - uL;
    if (ole<Ops>(h_min, drytol)) {
        if (REC) rec->rs = 0;
        hm = 0.0;
        double t = ((uR + uL) - oscale(sqR, 1, 2.0, o)) + oscale(sqL, 1, 2.0, o);
        s1m = t;
        s2m = t;
        return;
    }
    double F_min = delu + oscale(sq_min - sq_max, 1, 2.0, o);
    double F_max = 0.0;  // needed only when F_min <= 0
    if (!ogt0<Ops>(F_min)) F_max = delu + (h_max - h_min) * o.sqrt(o.div1((0.5 * g) * (h_max + h_min), h_max * h_min));
    if (ogt0<Ops>(F_min)) {  // two rarefactions
        const double t0 = -delu + oscale(sqL + sqR, 1, 2.0, o);
        double t = omax<Ops>(0.0, t0);
        if (REC) {
            rec->rs = 1;
            rec->t_pos = !olt<Ops>(t0, 0.0);
        }
        hm = (1.0 / (16.0 * g)) * (t * t);
        const double sqm = o.sqrt(g * hm);
        s1m = (uL + oscale(sqL, 1, 2.0, o)) - 3.0 * sqm;
        s2m = (uR - oscale(sqR, 1, 2.0, o)) + 3.0 * sqm;
    } else if (ole<Ops>(F_max, 0.0)) {  // two shocks: one Newton step on sqrt(h)
        if (REC) rec->rs = 2;
        const double h0 = h_max;
        double iL, iR, F0, dfdh;
        if (Ops::kFast) {
            // h0 is one side's depth, whose terms in F0 and dfdh are products of a zero
            // with a finite value: the other ("low") side's remain, in the order of
            // F0 = (delu + (h0 - hL) gL) + (h0 - hR) gR and
            // dfdh = ((gL - XL) + gR) - XR, X = g (h0 - h) / ((4 h0^2) g_side)
            const bool l_low = r_higher;
            const double hl = l_low ? hL : hR;
            const double i0 = o.div(1.0, l_low ? Recip{hR, yR} : Recip{hL, yL});
            const double il = o.div(1.0, l_low ? Recip{hL, yL} : Recip{hR, yR});
            const double g0 = o.sqrt((0.5 * g) * (i0 + i0)), gl = o.sqrt((0.5 * g) * (i0 + il));
            const double dl = h0 - hl;
            F0 = delu + dl * gl;
            const double xl = flip(o.div1(g * dl, (4.0 * (h0 * h0)) * gl), true);
            dfdh = ((l_low ? gl : g0) + (l_low ? xl : gl)) + (l_low ? g0 : xl);
            iL = l_low ? il : i0;
            iR = l_low ? i0 : il;
        } else {
            const double i0 = r_higher ? o.div(1.0, Recip{hR, yR}) : o.div(1.0, Recip{hL, yL});
            iL = o.div(1.0, Recip{hL, yL});
            iR = o.div(1.0, Recip{hR, yR});
            const double gL = o.sqrt((0.5 * g) * (i0 + iL)), gR = o.sqrt((0.5 * g) * (i0 + iR));
            F0 = (delu + (h0 - hL) * gL) + (h0 - hR) * gR;
            dfdh = ((gL - o.div1(g * (h0 - hL), (4.0 * (h0 * h0)) * gL)) + gR) -
                   o.div1(g * (h0 - hR), (4.0 * (h0 * h0)) * gR);
        }
        const double sq0 = o.sqrt(h0);
        double slope = oscale(sq0, 1, 2.0, o) * dfdh;
        double t = sq0 - o.div1(F0, slope);
        hm = t * t;
        const double im = o.div1(1.0, hm);
        double u1m = uL - (hm - hL) * o.sqrt((0.5 * g) * (im + iL));
        double u2m = uR + (hm - hR) * o.sqrt((0.5 * g) * (im + iR));
        const double sqm = o.sqrt(g * hm);
        s1m = u1m - sqm;
        s2m = u2m + sqm;
    } else {  // one shock, one rarefaction
        if (REC) {
            rec->rs = 3;
            rec->lhigh = olt<Ops>(hR, hL);
        }
        const double h0 = h_min;
        double F0 = F_min;  // + (h0 - h_min) sqrt(...), a zero while the root is finite
        if (!Ops::kFast) {
            const double i0 = r_lower ? o.div(1.0, Recip{hR, yR}) : o.div(1.0, Recip{hL, yL});
            F0 = F_min + (h0 - h_min) * o.sqrt((0.5 * g) * (i0 + i0));
        }
        double slope = o.div1(F_max - F0, h_max - h_min);
        hm = h0 - o.div1(F0, slope);
        const double sqm = o.sqrt(g * hm);
        if (olt<Ops>(hR, hL)) {
            s1m = (uL + oscale(sqL, 1, 2.0, o)) - 3.0 * sqm;
            s2m = (uL + oscale(sqL, 1, 2.0, o)) - sqm;
        } else {
            s2m = (uR - oscale(sqR, 1, 2.0, o)) + 3.0 * sqm;
            s1m = (uR - oscale(sqR, 1, 2.0, o)) + sqm;
        }
    }
}

// The middle depth riemanntype gives for a wet side against its own mirror image
// (depths h, h, velocities u, -u), the wet/dry edges' wall test; u points at the
// dry side, sq = sqrt(g h), y = recip_fix(h). With equal depths hm is the
// expressions' value with their zero factors gone: F_min and F_max are both
// delu = -u - u up to a signed zero, the wave is two rarefactions for delu > 0,
// else two shocks whose Newton step has F0 = delu and dfdh = gL + gR, gL = gR
// (each dropped term is a product of a zero with a finite value). One quotient
// and two roots instead of six quotients and seven roots: these edges stand alone
// in their warps, so their chain is the warp's (bowl of 2^12 cells: 40e3 cycles
// of the edge phase before, 11e3 without such edges). Depths outside
// recip_fix's range, whose products may not be finite, take the general form.
static __device__ __noinline__ double wall_depth(double h, double u, double sq, u64 y, double drytol) {
    if (y == 0) y = recip_fix(h);  // left out for a cell at rest
    if (y == 0) {
        double hm, s1m, s2m;
        SafeOps o;
        riemann_structure_rec<false>(h, h, u, -u, drytol, sq, sq, y, y, hm, s1m, s2m, nullptr, o);
        return hm;
    }
    const double delu = -u - u;
    double t;
    if (gt0(delu)) {
        t = imax(0.0, -delu + scale_pow2(sq + sq, 1, 2.0));
        return (1.0 / (16.0 * kG)) * (t * t);
    }
    const double i = div_fix(1.0, h, y);
    const double gL = sqrt_fix((0.5 * kG) * (i + i));
    const double sq0 = sqrt_fix(h);
    t = sq0 - div_one(delu, scale_pow2(sq0, 1, 2.0) * (gL + gL));
    return t * t;
}

__device__ __forceinline__ double det3(double a00, double a01, double a02, double a10, double a11, double a12,
                                       double a20, double a21, double a22) {
    double d1 = a00 * (a11 * a22 - a12 * a21);
    double d2 = a01 * (a10 * a22 - a12 * a20);
    double d3 = a02 * (a10 * a21 - a11 * a20);
    return (d1 - d2) + d3;
}

// RN(0 * x): a zero with x's sign for finite x (0 * inf and 0 * NaN are NaN).
__device__ __forceinline__ double mul0(double x) {
    return is_finite(x) ? bitsd(dbits(x) & (long long)0x8000000000000000ULL) : x * 0.0;
}
// |x| < 2^300 (or zero): products of three such numbers neither overflow nor are infinite
__device__ __forceinline__ bool moderate(double x) { return abs_bits(x) < 0x52b0000000000000LL; }

// Augmented solver (George 2008) with maxiter = 1, src/geoclaw/riemannsolvers.f:2-258.
// The entropy corrector is off in the source; with one iteration the star
// states after the Cramer solve never reach the outputs.
// sqL / sqR: sqrt(g * h) of the (fixed-up) depths; yL / yR: recip_fix of them (or 0).
//
// The 3x3 Cramer solve has the eigenvector matrix R = [[1, 0, 1], [l0, 0, l2],
// [l0^2, 1, l2^2]] with constant 0 and 1 entries. Evaluated in the source's
// order, a product by 1 is its other factor and a product by 0 a signed zero,
// and subtracting or adding a zero leaves a nonzero value unchanged, so for
// finite operands the four determinants have the values
//   det(R) = RN(l0 - l2), the numerators RN(e1 - RN(e0 l2)), the full
//   expression for beta1, and RN(RN(e0 l0) - e1)
// with at most a different sign of a zero result. Such a zero only reaches the
// f-waves, whose zeros the net-update accumulation turns into +0, except as a
// divisor: a zero determinant, and operands that are not finite or so large
// that a product could overflow, take the source's full expressions.
template <bool REC, class Ops>
__device__ __forceinline__ void riemann_aug_rec(double hL, double hR, double huL, double huR, double bL, double bR,
                                               double uL, double uR, double vL, double vR, double delphi,
                                               double sE1, double sE2, double sqL, double sqR, u64 yL,
                                               u64 yR, double drytol, double sw[3],
                                               double fw[3][3], AugRec* rec, Ops& o) {
    const double g = kG;
    double delh = hR - hL;
    double delhu = huR - huL;
    double delb = bR - bL;
    double hm, s1m, s2m;
    riemann_structure_rec<REC>(hL, hR, uL, uR, drytol, sqL, sqR, yL, yR, hm, s1m, s2m, rec, o);
    double l0 = omin<Ops>(sE1, s2m);
    double l2 = omax<Ops>(sE2, s1m);
    if (REC) {
        rec->l0_sE1 = olt<Ops>(sE1, s2m);
        rec->l2_sE2 = olt<Ops>(s1m, sE2);
        rec->s1m = s1m;
        rec->s2m = s2m;
    }
    sE1 = l0;
    sE2 = l2;
    // sE2 - sE1 = -(l0 - l2) exactly (round to nearest is symmetric): one
    // reciprocal serves hstarHLL's divisor and the Cramer determinant
    const double dsp = sE2 - sE1;
    const Recip rsp = recip_of(dsp);
    const double hq = o.div(((huL - huR) + sE2 * hR) - sE1 * hL, rsp);
    double hstarHLL = omax<Ops>(hq, 0.0);
    double l1 = oscale(l0 + l2, -1, 0.5, o);
    if (olt<Ops>(iabs(l1), 1e-20)) l1 = 0.0;
    const double r20 = l0 * l0, r22 = l2 * l2;

    const double ct = 1e-6;
    const double hhalf = oscale(hL + hR, -1, 0.5, o);
    double hbar = omax<Ops>(hhalf, 0.0);
    double su = uL + uR;
    const double ghbar = g * hbar;
    double s1s2bar = oscale(su * su, -2, 0.25, o) - ghbar;
    const double uLR = uL * uR;
    double s1s2tilde = omax<Ops>(0.0, uLR) - ghbar;
    bool sonic = ole<Ops>(iabs(s1s2bar), ct);
    sonic |= ole<Ops>(s1s2bar * s1s2tilde, ct);
    sonic |= ole<Ops>((s1s2bar * sE1) * sE2, ct);
    sonic |= olt<Ops>(omin<Ops>(iabs(sE1), iabs(sE2)), ct);
    sonic |= olt0<Ops>(sE1) & ogt0<Ops>(s1m);
    sonic |= ogt0<Ops>(sE2) & olt0<Ops>(s2m);
    sonic |= olt0<Ops>((uL + sqL) * (uR + sqR));  // sqrt(g * h) of the fixed-up depths
    sonic |= olt0<Ops>((uL - sqL) * (uR - sqR));
    if (REC) {
        rec->hst_pos = olt<Ops>(0.0, hq);
        rec->hbar_pos = olt<Ops>(0.0, hhalf);
        rec->tilde_x = !olt<Ops>(uLR, 0.0);
        rec->sonic = sonic;
        rec->dcase = 0;
    }

    const double dgh = (delb * g) * hbar;
    const double qh = o.div1_if(!sonic, dgh, s1s2bar);
    const double qphi = flip(o.div1_if(!sonic, dgh * s1s2tilde, s1s2bar), true);
    double deldelh = sonic ? flip(delb, true) : qh;
    double deldelphi = sonic ? flip(ghbar * delb, true) : qphi;
    const double hsd = hstarHLL * dsp;
    const bool apart = olt<Ops>(sE1, -ct) & olt<Ops>(ct, sE2);
    const int dcase = apart ? 1 : (ole<Ops>(ct, sE1) ? 2 : (ole<Ops>(sE2, -ct) ? 3 : 0));
    // the two bounds of the case, without a branch per case
    const double q1 = o.div1_if((dcase == 1) | (dcase == 2), hsd, sE1), q2 = o.div1_if((dcase == 1) | (dcase == 3), hsd, sE2);
    const double hi = dcase == 1 ? q2 : (dcase == 2 ? q1 : hR);
    const double lo = dcase == 1 ? q1 : (dcase == 2 ? flip(hL, true) : q2);
    const double x1 = omin<Ops>(deldelh, hi);
    if (REC && dcase) {
        rec->dcase = (int8_t)dcase;
        rec->dd_min_first = olt<Ops>(deldelh, hi);
        rec->dd_max_first = olt<Ops>(lo, x1);
    }
    deldelh = dcase ? omax<Ops>(x1, lo) : deldelh;
    const double pl = flip(hL * delb, true), pr = flip(hR * delb, true);
    const double gmx = g * omax<Ops>(pl, pr), gmn = g * omin<Ops>(pl, pr);
    const double y1 = omin<Ops>(deldelphi, gmx);
    if (REC) {
        rec->ph_mx_pl = olt<Ops>(pr, pl);
        rec->ph_min_first = olt<Ops>(deldelphi, gmx);
        rec->ph_mn_pl = olt<Ops>(pl, pr);
        rec->ph_max_first = olt<Ops>(gmn, y1);
    }
    deldelphi = omax<Ops>(y1, gmn);
    double d0 = delh - deldelh, d1 = delhu, d2 = delphi - deldelphi;

    double beta0 = 0.0, beta1 = 0.0, beta2 = 0.0;
    const double det = l0 - l2;
    const bool quick = moderate(l0) & moderate(l2) & moderate(d0) & moderate(d1) & moderate(d2) &
                       ((dbits(det) << 1) != 0);
    // beta1's numerator, the source's expression with the products by 1 dropped
    const double n1 = ((d1 * r22 - l2 * d2) - d0 * (l0 * r22 - l2 * r20)) + (l0 * d2 - d1 * r20);
    if (Ops::kFast || quick) {
        o.ok = o.ok & quick;
        const Recip rd{det, rsp.y};  // det = -(sE2 - sE1): the same significand
        beta0 = o.div(d1 - d0 * l2, rd);
        beta1 = o.div(n1, rd);
        beta2 = o.div(d0 * l0 - d1, rd);
    } else if (!Ops::kFast) {
        const double r00 = 1.0, r01 = 0.0, r02 = 1.0, r10 = l0, r11 = 0.0, r12 = l2, r21 = 1.0;
        const double dt = det3(r00, r01, r02, r10, r11, r12, r20, r21, r22);
        beta0 = det3(d0, r01, r02, d1, r11, r12, d2, r21, r22) / dt;
        beta1 = det3(r00, d0, r02, r10, d1, r12, r20, d2, r22) / dt;
        beta2 = det3(r00, r01, d0, r10, r11, d1, r20, r21, d2) / dt;
    }

    sw[0] = l0;
    sw[1] = l1;
    sw[2] = l2;
    // f-waves: beta times rows 2 and 3 of R (r11 = 0, r21 = 1)
    fw[0][0] = beta0 * l0; fw[1][0] = beta0 * r20; fw[2][0] = (beta0 * l0) * vL;
    fw[0][1] = Ops::kFast ? bitsd(dbits(beta1) & (long long)0x8000000000000000ULL) : mul0(beta1); fw[1][1] = beta1;
    fw[0][2] = beta2 * l2; fw[1][2] = beta2 * r22; fw[2][2] = (beta2 * l2) * vR;
    fw[2][1] = ((((hR * uR) * vR) - ((hL * uL) * vL)) - fw[2][0]) - fw[2][2];
}

// Wet/dry handling, wave speeds and net updates of c_bind_geoclaw_solver_dp
// (src/geoclaw/c_bind_riemannsolvers.f90:16-176) with the f-wave
// (src/geoclaw/riemannsolvers.f:446-500) or augmented solver. netL/netR are
// the left/right net updates of (h, hu, hv) in the edge frame.
// sqL0 / sqR0 are sqrt(g * depth) of the two cells, computed once per cell by the
// caller; they are used only where the reference evaluates sqrt(g * h) on an
// unmodified wet depth (the same operands, so the same bits).
// yL0 / yR0 are recip_fix of the two depths (0 for a dry side, or left out where the
// side's momenta are zeros).
// Branch-frozen evaluation (FZ, the f-wave only): FZ = 1 records the decisions
// of the edge into *fz, FZ = 2 takes them from *fz instead of the comparisons
// (a forward run whose every branch is that of a recorded run, for checking the
// discrete adjoint by finite differences). Bits: 0 both sides dry, 1 right wet,
// 2 left wet, 3 right wall, 4 right bottom lowered, 5 left wall, 6 left bottom
// lowered, 7 sE1 = sL, 8 sE2 = sR, 9 + 2w / 10 + 2w wave w's speed < 0 / > 0.
template <int FZ>
__device__ __forceinline__ bool fzb(uint16_t* fz, int bit, bool v) {
    if (FZ == 2) return (*fz >> bit) & 1u;
    if (FZ == 1 && v) *fz |= (uint16_t)(1u << bit);
    return v;
}

template <int SOLVER, int FZ, class Ops>
__device__ __forceinline__ void geoclaw_solver(double hL, double hR, double huL, double huR, double hvL,
                                               double hvR, double bL, double bR, double sqL0, double sqR0,
                                               u64 yL0, u64 yR0, double drytol, double netL[3],
                                               double netR[3], double& maxspeed, uint16_t* fz, Ops& o) {
    const double g = kG;
    netL[0] = netL[1] = netL[2] = 0.0;
    netR[0] = netR[1] = netR[2] = 0.0;
    maxspeed = 0.0;
    if (FZ == 1) *fz = 0;
    const bool wetR0 = fzb<FZ>(fz, 1, lt(drytol, hR)), wetL0 = fzb<FZ>(fz, 2, lt(drytol, hL));  // h > drytol
    if (fzb<FZ>(fz, 0, !wetL0 && !wetR0 && !is_nan(hL) && !is_nan(hR) && !is_nan(drytol))) return;  // both dry
    if (FZ == 2) {  // a recorded wet side is wet here, whatever its current depth
        if (wetL0) sqL0 = sqrt_fix(g * hL);
        if (wetR0) sqR0 = sqrt_fix(g * hR);
    }
    double uL, uR, vL, vR;
    if (FZ == 2) {
        uR = wetR0 ? huR / hR : 0.0;
        vR = wetR0 ? hvR / hR : 0.0;
        uL = wetL0 ? huL / hL : 0.0;
        vL = wetL0 ? hvL / hL : 0.0;
    } else {
        const Recip rL{hL, yL0}, rR{hR, yR0};
        uR = o.div_if(wetR0, huR, rR);
        vR = o.div_if(wetR0, hvR, rR);
        uL = o.div_if(wetL0, huL, rL);
        vL = o.div_if(wetL0, hvL, rL);
    }
    if (!wetR0) {
        hR = 0.0; huR = 0.0; hvR = 0.0; uR = 0.0; vR = 0.0;
    }
    if (!wetL0) {
        hL = 0.0; huL = 0.0; hvL = 0.0; uL = 0.0; vL = 0.0;
    }
    // A dry side is a wall where the wet side's water cannot reach its bottom (wall(1)
    // = 0 resp. wall(3) = 0, wall(2) = 0 with either), else its bottom is lowered to
    // the wet side's surface. Both orientations in one block: each of its parts is a
    // chain of its own for the warp.
    bool wall_l = false, wall_r = false;
    if (!(wetL0 & wetR0)) {
        const bool rdry = !wetR0;  // hR is now 0.0, and 0.0 <= drytol
        const double h = rdry ? hL : hR, u = rdry ? uL : -uR, b = rdry ? bL : bR, bd = rdry ? bR : bL;
        const double hstar = FZ != 2 ? wall_depth(h, u, rdry ? sqL0 : sqR0, rdry ? yL0 : yR0, drytol) : 0.0;
        const double low = h + b;
        const bool wall = fzb<FZ>(fz, rdry ? 3 : 5, lt(imax(h, hstar) + b, bd));
        const bool lower = wall ? false : fzb<FZ>(fz, rdry ? 4 : 6, lt(low, bd));
        wall_r = wall && rdry;
        wall_l = wall && !rdry;
        if (wall_r) {
            hR = hL; huR = -huL; bR = bL; uR = -uL; vR = vL;
        }
        if (wall_l) {
            hL = hR; huL = -huR; bL = bR; uL = -uR; vL = vR;
        }
        bR = lower && rdry ? low : bR;
        bL = lower && !rdry ? low : bL;
    }
    const double hsum = hR + hL;
    const double ghalf_h = prod(g * 0.5, hsum);  // (0.5 * g) * (hR + hL): delphi, chat, the f-wave's deldelphi
    double delphi = ((prod(huR - huL, uL + uR) - prod(prod(uL, uR), hR - hL)) +
                     prod(prod(0.5 * g, ((bR + hR) - bL) - hL), hsum)) -
                    prod(ghalf_h, bR - bL);
    // sqrt(g * h) after the wet/dry fix-ups: a wet side keeps its depth, a dry one
    // has depth 0, and a wall mirrors the wet side's depth
    // a dry side has h = 0 <= drytol now, a wet one is unchanged, a wall mirrors the wet side
    const bool wetL = wetL0 || wall_l, wetR = wetR0 || wall_r;
    double sqL = wetL ? (wall_l ? sqR0 : sqL0) : 0.0;
    double sqR = wetR ? (wall_r ? sqL0 : sqR0) : 0.0;
    double sL = uL - sqL;
    double sR = uR + sqR;
    double uhat = o.div1(prod(sqL, uL) + prod(sqR, uR), sqR + sqL);
    double chat = o.sqrt(ghalf_h);
    const double r1 = uhat - chat, r2 = uhat + chat;
    double sE1 = fzb<FZ>(fz, 7, olt<Ops>(sL, r1)) ? sL : r1;  // imin(sL, r1)
    double sE2 = fzb<FZ>(fz, 8, olt<Ops>(r2, sR)) ? sR : r2;  // imax(sR, r2)

    double sw[3], fw[3][3];
    if (SOLVER == AUG_RIEMANN) {
        // the reciprocals of the fixed-up depths: a wet side's own, a wall's mirrored one
        const u64 yLf = wall_l ? yR0 : yL0, yRf = wall_r ? yL0 : yR0;
        riemann_aug_rec<false>(hL, hR, huL, huR, bL, bR, uL, uR, vL, vR, delphi, sE1, sE2, sqL, sqR, yLf, yRf, drytol, sw,
                               fw, nullptr, o);
    } else {
        double delhu = huR - huL;
        double delb = bR - bL;
        double deldelphi = -prod(ghalf_h, delb);
        double dpd = delphi - deldelphi;
        const Recip rD = recip_of(sE2 - sE1);
        double beta1 = o.div(prod(sE2, delhu) - dpd, rD);
        double beta2 = o.div(dpd - prod(sE1, delhu), rD);
        // Of the middle speed (sE1 + sE2) / 2 the net updates read the sign, which is the
        // exact sum's (a sum of doubles rounds to zero only where it is zero, and with sE2 -
        // sE1 in the reciprocal's range halving it does not underflow), and the maximum
        // never takes it: half a rounded sum is at most the larger of the two magnitudes.
        const long long k1 = num_key(sE1), k2 = num_key(flip(sE2, true));
        const double sign = k1 < k2 ? -1.0 : (k1 > k2 ? 1.0 : 0.0);
        sw[0] = sE1; sw[1] = Ops::kFast ? sign : scale_pow2(sE1 + sE2, -1, 0.5); sw[2] = sE2;
        fw[0][0] = beta1; fw[1][0] = prod(beta1, sE1); fw[2][0] = prod(beta1, vL);
        fw[0][2] = beta2; fw[1][2] = prod(beta2, sE2); fw[2][2] = prod(beta2, vR);
        fw[0][1] = 0.0; fw[1][1] = 0.0;
        fw[2][1] = ((prod(huR, vR) - prod(huL, vL)) - fw[2][0]) - fw[2][2];
    }
    // eliminate ghost fluxes of a wall: multiplication by 0, i.e. zeros whose signs the
    // net updates drop, except for values that are not finite
#pragma unroll
    for (int w = 0; w < 3; ++w) {
        const bool gone = (wall_l & (w < 2)) | (wall_r & (w > 0));
        if (Ops::kFast) {
            o.ok = o.ok & (!gone | (is_finite(sw[w]) & is_finite(fw[0][w]) & is_finite(fw[1][w]) & is_finite(fw[2][w])));
            sw[w] = gone ? 0.0 : sw[w];
            fw[0][w] = gone ? 0.0 : fw[0][w];
            fw[1][w] = gone ? 0.0 : fw[1][w];
            fw[2][w] = gone ? 0.0 : fw[2][w];
        } else if (gone) {
            sw[w] = sw[w] * 0.0;
            fw[0][w] = fw[0][w] * 0.0;
            fw[1][w] = fw[1][w] * 0.0;
            fw[2][w] = fw[2][w] * 0.0;
        }
    }
    // net updates: each accumulator starts at +0 and takes its waves in wave order;
    // +0 + x is z0(x), and the f-wave's wave 2 carries exact +0 in h and hu,
    // which leaves an accumulator unchanged (it is never -0)
    const bool neg1 = olt0<Ops>(sw[1]);
    const bool sub = (FZ == 0) & olt0<Ops>(sw[0]) & ogt0<Ops>(sw[2]) & (neg1 | ogt0<Ops>(sw[1]));
    // subcritical flow, as almost everywhere: wave 0 goes left, wave 2 right, the
    // middle one to one side, in one sum and without branches
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const double f0 = z0(fw[e][0]), f2 = fw[e][2];
        if (FZ != 0) continue;
        if (SOLVER != AUG_RIEMANN && e < 2) {
            netL[e] = f0;
            netR[e] = z0(f2);
        } else {
            const double sum = (neg1 ? f0 : z0(fw[e][1])) + (neg1 ? fw[e][1] : f2);
            netL[e] = neg1 ? sum : f0;
            netR[e] = neg1 ? z0(f2) : sum;
        }
    }
    SWE_IF(!sub) {
        bool tL[3] = {false, false, false}, tR[3] = {false, false, false};
        auto acc = [](double& a, bool& t, double c) {
            a = t ? a + c : z0(c);
            t = true;
        };
#pragma unroll
        for (int e = 0; e < 3; ++e) netL[e] = netR[e] = 0.0;
#pragma unroll
        for (int w = 0; w < 3; ++w) {
            const bool neg = fzb<FZ>(fz, 9 + 2 * w, olt0<Ops>(sw[w])), pos = fzb<FZ>(fz, 10 + 2 * w, ogt0<Ops>(sw[w]));
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                if (SOLVER != AUG_RIEMANN && w == 1 && e < 2) continue;
                const double f = fw[e][w];
                if (neg) {
                    acc(netL[e], tL[e], f);
                } else if (pos) {
                    acc(netR[e], tR[e], f);
                } else {
                    const double hf = 0.5 * f;
                    acc(netL[e], tL[e], hf);
                    acc(netR[e], tR[e], hf);
                }
            }
        }
    }
    // m = |s1|; if (|s2| > m) m = |s2|; if (|s3| > m) m = |s3|, on the bit
    // patterns (non-negative values order like them; a NaN candidate never wins)
    long long m = abs_bits(sw[0]);
    const long long a1 = abs_bits(sw[1]), a2 = abs_bits(sw[2]);
    if (Ops::kFast ? SOLVER == AUG_RIEMANN && a1 > m : a1 > m && not_nan(a1)) m = a1;
    if (a2 > m && (Ops::kFast || not_nan(a2))) m = a2;
    maxspeed = bitsd(m);
}

// compute_geoclaw_flux, src/SWE/SWE_euler_timestep.f90:449-481.
// axis: 0 = any normal; 1 = n = (+-1, +0); 2 = n = (+0, +-1). For an
// axis-aligned normal each component of T p and of net(2:3) T is one exact
// product plus a signed zero, i.e. the other momentum with its sign flipped
// and -0 mapped to +0, which integer instructions give bit for bit while the
// operands are finite (0 * inf would be NaN). For a diagonal normal
// (|n1| = |n2| = c) the four products of each rotation are +-RN(c p1) and
// +-RN(c p2), since RN(-x) = -RN(x): two products per side, the signs set on
// the bit patterns. Otherwise the general form runs.
template <int SOLVER, int FZ, class Ops>
__device__ __forceinline__ void geoclaw_rotated(double n1, double n2, const State& QL, const State& QR, double dL,
                                                double dR, double sqL, double sqR, u64 yL, u64 yR, double drytol,
                                                Update& fL, Update& fR, int axis, uint16_t* fz, Ops& o) {
    const bool fin = is_finite(QL.p1) & is_finite(QL.p2) & is_finite(QR.p1) & is_finite(QR.p2);
    const bool fast = (axis != 0) & fin;
    const bool diag = (axis == 0) & fin & (abs_bits(n1) == abs_bits(n2));
    const bool sn = axis == 1 ? lt0(n1) : lt0(n2);  // sign of the nonzero component
    const bool g1 = dbits(n1) < 0, g2 = dbits(n2) < 0;  // sign bits of the normal
    const double c = bitsd(abs_bits(n1));
    // FastOps takes the mesh's normals and finite momenta
    o.ok = o.ok & (!Ops::kFast | diag | fast);
    // axis-aligned; for a diagonal or a general normal overwritten below
    const bool ax1 = axis == 1;
    double pL1 = z0(flip(ax1 ? QL.p1 : QL.p2, sn)), pL2 = z0(flip(ax1 ? QL.p2 : QL.p1, ax1 ? sn : !sn));
    double pR1 = z0(flip(ax1 ? QR.p1 : QR.p2, sn)), pR2 = z0(flip(ax1 ? QR.p2 : QR.p1, ax1 ? sn : !sn));
    SWE_IF(diag) {
        // RN(n1 p1) = +-a1, RN(n2 p2) = +-a2, RN(-n2 p1) = -+a1, RN(n1 p2) = +-a2
        const double aL1 = prod_rot(c, QL.p1), aL2 = prod_rot(c, QL.p2);
        const double aR1 = prod_rot(c, QR.p1), aR2 = prod_rot(c, QR.p2);
        pL1 = z0(flip(aL1, g1)) + flip(aL2, g2);
        pL2 = z0(flip(aL1, !g2)) + flip(aL2, g1);
        pR1 = z0(flip(aR1, g1)) + flip(aR2, g2);
        pR2 = z0(flip(aR1, !g2)) + flip(aR2, g1);
    }
    if (!Ops::kFast && !diag && !fast) {
        // T = [[n1, n2], [-n2, n1]]; p_edge = T p
        pL1 = z0(prod_rot(n1, QL.p1)) + prod_rot(n2, QL.p2);
        pL2 = z0(prod_rot(-n2, QL.p1)) + prod_rot(n1, QL.p2);
        pR1 = z0(prod_rot(n1, QR.p1)) + prod_rot(n2, QR.p2);
        pR2 = z0(prod_rot(-n2, QR.p1)) + prod_rot(n1, QR.p2);
    }
    double netL[3], netR[3], ms;
    geoclaw_solver<SOLVER, FZ>(dL, dR, pL1, pR1, pL2, pR2, QL.b, QR.b, sqL, sqR, yL, yR, drytol, netL, netR, ms, fz,
                               o);
    fL.h = netL[0];
    fL.s = ms;
    fR.h = netR[0];
    fR.s = ms;
    const bool nfin = is_finite(netL[1]) & is_finite(netL[2]) & is_finite(netR[1]) & is_finite(netR[2]);
    o.ok = o.ok & (!Ops::kFast | nfin);
    fL.p1 = z0(flip(ax1 ? netL[1] : netL[2], ax1 ? sn : !sn)); fL.p2 = z0(flip(ax1 ? netL[2] : netL[1], sn));
    fR.p1 = z0(flip(ax1 ? netR[1] : netR[2], ax1 ? sn : !sn)); fR.p2 = z0(flip(ax1 ? netR[2] : netR[1], sn));
    SWE_IF(diag && (Ops::kFast || nfin)) {
        // RN(m1 n1) = +-b1, RN(m2 (-n2)) = -+b2, RN(m1 n2) = +-b1, RN(m2 n1) = +-b2
        const double bL1 = prod_rot(netL[1], c), bL2 = prod_rot(netL[2], c);
        const double bR1 = prod_rot(netR[1], c), bR2 = prod_rot(netR[2], c);
        fL.p1 = z0(flip(bL1, g1)) + flip(bL2, !g2);
        fL.p2 = z0(flip(bL1, g2)) + flip(bL2, g1);
        fR.p1 = z0(flip(bR1, g1)) + flip(bR2, !g2);
        fR.p2 = z0(flip(bR1, g2)) + flip(bR2, g1);
    }
    if (!Ops::kFast && (!nfin || (!diag && !fast))) {
        // p = net(2:3) T
        fL.p1 = z0(prod_rot(netL[1], n1)) + prod_rot(netL[2], -n2);
        fL.p2 = z0(prod_rot(netL[1], n2)) + prod_rot(netL[2], n1);
        fR.p1 = z0(prod_rot(netR[1], n1)) + prod_rot(netR[2], -n2);
        fR.p2 = z0(prod_rot(netR[1], n2)) + prod_rot(netR[2], n1);
    }
}

// SURFACE: the states' h is the surface (else the depth, and not read).
template <int SOLVER, int FZ, bool SURFACE, class Ops>
__device__ __forceinline__ void geoclaw_flux(double n1, double n2, const State& QL, const State& QR, double dL,
                                             double dR, double sqL, double sqR, u64 yL, u64 yR,
                                             double drytol, Update& fL, Update& fR, int axis, uint16_t* fz, Ops& o) {
    // both sides dry: the solver returns zero net updates and speed, and their
    // rotation back is +0 in every component, so neither rotation is needed
    // (the tests of these branches are joined with & and |: a short-circuit test is a
    // chain of branches, and lanes that leave it at different tests stay apart for
    // the whole solver, which the warp then runs twice)
    const bool dry2 = FZ == 2 ? ((*fz & 1u) != 0)
                              : !(lt(drytol, dL) | lt(drytol, dR) | is_nan(dL) | is_nan(dR) | is_nan(drytol));
    bool rest = false;
    if (SOLVER == FWAVE && FZ == 0) {
        // Water at rest on both sides under one surface (lake at rest): every
        // momentum is +-0, both sides are wet and the c-binding's surface
        // difference ((bR + hR) - bL) - hL is +-0. Then in the f-wave path the
        // velocities, uhat and the momentum jump are signed zeros; delphi is
        // +-0 - X with X = RN(ghalf_h (bR - bL)) and deldelphi is -X, so
        // delphi - deldelphi is a zero (x - x = +0), both f-wave coefficients
        // divide a zero, and every f-wave component is a signed zero. The net
        // updates start at +0 and add zeros, so they are +0, and rotating them
        // back gives +0 in every component. The speeds are sL = -sqL,
        // sR = sqR, Roe uhat -+ chat = -+chat with chat = sqrt(ghalf_h), so
        // |sE1| = max(sqL, chat), |sE2| = max(sqR, chat), and the middle wave's
        // |RN(sE1 + sE2) / 2| (sE1 <= 0 <= sE2) exceeds neither: the maximum
        // speed is the largest of sqL, sqR and chat. And chat never exceeds
        // the larger of sqL, sqR: with h the larger depth, RN(hR + hL) <= 2h,
        // so ghalf_h = RN(RN(g / 2) RN(hR + hL)) <= RN((g / 2) 2h) = RN(g h)
        // (g / 2 is exact, and RN, the product by a positive factor and sqrt
        // are monotone), hence chat <= RN(sqrt(RN(g h))), the cell's own
        // sqrt(g h). So the maximum speed is max(sqL, sqR), both positive. The
        // same bits as the full evaluation, without its FP64 arithmetic.
        // The surface difference x - hL, x = RN(RN(bR + hR) - bL), rounds to a
        // zero exactly when x equals hL and both are finite (gradual underflow:
        // the difference of two distinct finite doubles is not rounded to zero;
        // inf - inf is NaN). hL > drytol >= 0 is positive, so equal values have
        // equal bit patterns: one FP64 addition fewer per edge.
        const bool still = ((dbits(QL.p1) | dbits(QL.p2) | dbits(QR.p1) | dbits(QR.p2)) << 1) == 0;
        // Where both surfaces are at +-0 (the sea level), dL = -bL and dR = -bR
        // exactly, so x = 0 - bL = dL for finite depths: no FP64 arithmetic at all. Only
        // where the surfaces are at hand (SURFACE): the step kernel on device-resident
        // states keeps the depths in their place, and asking their bits against the
        // bathymetry's instead costs more than the two additions (basin of 2^24 cells, 4
        // steps: 4366 us against 4315).
        const bool can = still & lt(drytol, dL) & lt(drytol, dR) & is_finite(dL) & is_finite(dR);
        const bool level = SURFACE && ((dbits(QL.h) | dbits(QR.h)) << 1) == 0;
        rest = can & level;
        SWE_IF(can & !level) rest = dbits((QR.b + dR) - QL.b) == dbits(dL);
    }
    if (dry2 | rest) {
        if (FZ == 1) *fz = 1;
        const double ms = rest ? bitsd(dbits(sqL) > dbits(sqR) ? dbits(sqL) : dbits(sqR)) : 0.0;
        fL = Update{0.0, 0.0, 0.0, ms};
        fR = Update{0.0, 0.0, 0.0, ms};
    } else {
        geoclaw_rotated<SOLVER, FZ>(n1, n2, QL, QR, dL, dR, sqL, sqR, yL, yR, drytol, fL, fR, axis, fz, o);
    }
}

// z0(n1 (p1 / d)) + n2 (p2 / d), r = {d, recip_fix(d)}
template <class Ops>
__device__ __forceinline__ double normal_velocity(double n1, double n2, double p1, double p2, const Recip& r, Ops& o) {
    return z0(n1 * o.div(p1, r)) + n2 * o.div(p2, r);
}

// lf_flux of two sides at or above the dry tolerance (the fluxes with bathymetry) for
// the mesh's normals, in 33 (axis-aligned) or 44 (diagonal) FP64 instructions instead
// of 49: a product with a component +-1 is a sign, one with +-0 a signed zero, whose
// addition only decides the sign of a zero sum (add_zero); the products of one value
// with the two components of a diagonal normal differ in sign; halves are exponents.
// `on` is the component along an axis-aligned normal, `off` the other one. For FastOps:
// other normals and values that are not finite leave o.ok false.
template <int SOLVER, class Ops>
__device__ __forceinline__ void lf_bath_wet(double n1, double n2, const State& QL, const State& QR, double hL,
                                            double hR, double cL, double cR, const Recip& rL, const Recip& rR,
                                            Update& fL, Update& fR, int axis, Ops& o) {
    const double g = kG;
    const bool second = axis == 2, diag = axis == 0;
    const double non = second ? n2 : n1, noff = second ? n1 : n2;
    const bool gon = dbits(non) < 0, goff = dbits(noff) < 0;
    const double pLon = second ? QL.p2 : QL.p1, pLoff = second ? QL.p1 : QL.p2;
    const double pRon = second ? QR.p2 : QR.p1, pRoff = second ? QR.p1 : QR.p2;
    const double pr = (0.5 * g) * (hL * hL + hR * hR);
    const double src = ((0.25 * g) * (hL + hR)) * (QR.b - QL.b);
    const double qL = o.div(pLon, rL), qR = o.div(pRon, rR);
    // (the off-axis quotients are finite, so their products with +-0 are zeros)
    auto bounded = [](double x) { return abs_bits(x) < 1524ll << 52; };
    o.ok = o.ok & is_finite(pr) & is_finite(src) & bounded(pLoff) & bounded(pRoff) &
           (!diag | (abs_bits(n1) == abs_bits(n2)));
    const u64 sign = 0x8000000000000000ull;
    double vL = z0(flip(qL, gon)), vR = z0(flip(qR, gon));
    double pon = flip(pr, gon), poff = bitsd((dbits(pr) ^ dbits(noff)) & (long long)sign);
    double son = flip(src, gon), soff = bitsd((dbits(src) ^ dbits(noff)) & (long long)sign);
    SWE_IF(diag) {
        const double c = iabs(n1);
        vL = z0(flip(c * qL, gon)) + flip(c * o.div(pLoff, rL), goff);
        vR = z0(flip(c * qR, gon)) + flip(c * o.div(pRoff, rR), goff);
        const double cp = c * pr, cs = c * src;
        pon = flip(cp, gon);
        poff = flip(cp, goff);
        son = flip(cs, gon);
        soff = flip(cs, goff);
    }
    fL.s = cL + iabs(vL);
    fR.s = cR + iabs(vR);
    const double alpha = (SOLVER == LLF_BATH) ? omax<Ops>(fL.s, fR.s) : 100.0;
    fL.h = oscale((hL * vL + hR * vR) + alpha * (QL.h - QR.h), -1, 0.5, o);
    fR.h = flip(fL.h, true);
    const double aon = pLon * vL + pRon * vR, aoff = pLoff * vL + pRoff * vR;
    double boff = add_zero(aoff, poff);
    SWE_IF(diag) boff = aoff + poff;
    const double fon = oscale((aon + pon) + alpha * (pLon - pRon), -1, 0.5, o);
    const double foff = oscale(boff + alpha * (pLoff - pRoff), -1, 0.5, o);
    const double lon = fon + son, ron = flip(fon, true) + son;
    double loff = add_zero(foff, soff), roff = add_zero(flip(foff, true), soff);
    SWE_IF(diag) {
        loff = foff + soff;
        roff = flip(foff, true) + soff;
    }
    fL.p1 = second ? loff : lon;
    fL.p2 = second ? lon : loff;
    fR.p1 = second ? roff : ron;
    fR.p2 = second ? ron : roff;
}

// compute_lf_flux, src/SWE/SWE_euler_timestep.f90:359-446
// sqL / sqR, yL / yR: sqrt(g * depth) and recip_fix of the two depths where they are
// above the dry tolerance (else not read).
template <int SOLVER, class Ops>
__device__ __forceinline__ void lf_flux(double n1, double n2, const State& QL, const State& QR, double dL,
                                        double dR, double drytol, Update& fL, Update& fR, double sqL,
                                        double sqR, u64 yL, u64 yR, int axis, Ops& o) {
    const double g = kG;
    if (SOLVER == LF_BATH || SOLVER == LLF_BATH) {
        const bool aL = lt(drytol, dL), aR = lt(drytol, dR);
        const Recip rL{dL, aL ? yL : recip_fix(dL)}, rR{dR, aR ? yR : recip_fix(dR)};
        const bool dryL = lt(dL, drytol), dryR = lt(dR, drytol);
        if (dryL || dryR) {
            fL = Update{0.0, 0.0, 0.0, 0.0};
            fR = Update{0.0, 0.0, 0.0, 0.0};
            SWE_IF(dryL && !dryR) {
                double hR = imax(dR, 0.0);
                double vR = normal_velocity(n1, n2, QR.p1, QR.p2, rR, o);
                fR.s = (aR ? sqR : o.sqrt(g * hR)) + iabs(vR);
                double pr = ((0.5 * g) * hR) * hR;
                fR.p1 = (-((0.5 * vR) * QR.p1) - pr * n1) + (0.5 * fR.s) * QR.p1;
                fR.p2 = (-((0.5 * vR) * QR.p2) - pr * n2) + (0.5 * fR.s) * QR.p2;
            }
            SWE_IF(dryR && !dryL) {
                double hL = imax(dL, 0.0);
                double vL = normal_velocity(n1, n2, QL.p1, QL.p2, rL, o);
                fL.s = (aL ? sqL : o.sqrt(g * hL)) + iabs(vL);
                double pr = ((0.5 * g) * hL) * hL;
                fL.p1 = ((0.5 * vL) * QL.p1 + pr * n1) + (0.5 * fL.s) * QL.p1;
                fL.p2 = ((0.5 * vL) * QL.p2 + pr * n2) + (0.5 * fL.s) * QL.p2;
            }
            return;
        }
        double hL = imax(dL, 0.0), hR = imax(dR, 0.0);
        double cL = sqL, cR = sqR;
        SWE_IF(!aL || !aR) {  // a depth at the tolerance
            cL = aL ? sqL : sqrt_fix(g * hL);
            cR = aR ? sqR : sqrt_fix(g * hR);
        }
        if (Ops::kFast) {
            lf_bath_wet<SOLVER>(n1, n2, QL, QR, hL, hR, cL, cR, rL, rR, fL, fR, axis, o);
            return;
        }
        double vL = normal_velocity(n1, n2, QL.p1, QL.p2, rL, o);
        double vR = normal_velocity(n1, n2, QR.p1, QR.p2, rR, o);
        fL.s = cL + iabs(vL);
        fR.s = cR + iabs(vR);
        double alpha = (SOLVER == LLF_BATH) ? imax(fL.s, fR.s) : 100.0;
        fL.h = 0.5 * ((hL * vL + hR * vR) + alpha * (QL.h - QR.h));
        fR.h = -fL.h;
        double pr = (0.5 * g) * (hL * hL + hR * hR);
        fL.p1 = 0.5 * (((QL.p1 * vL + QR.p1 * vR) + pr * n1) + alpha * (QL.p1 - QR.p1));
        fL.p2 = 0.5 * (((QL.p2 * vL + QR.p2 * vR) + pr * n2) + alpha * (QL.p2 - QR.p2));
        fR.p1 = -fL.p1;
        fR.p2 = -fL.p2;
        double src = ((0.25 * g) * (hL + hR)) * (QR.b - QL.b);
        fL.p1 = fL.p1 + src * n1;
        fL.p2 = fL.p2 + src * n2;
        fR.p1 = fR.p1 + src * n1;
        fR.p2 = fR.p2 + src * n2;
    } else {
        dL = QL.h - 0.0;
        dR = QR.h - 0.0;
        double hL = imax(dL, 0.0), hR = imax(dR, 0.0);
        double vL = normal_velocity(n1, n2, QL.p1, QL.p2, recip_of(dL), o);
        double vR = normal_velocity(n1, n2, QR.p1, QR.p2, recip_of(dR), o);
        fL.s = o.sqrt(g * dL) + iabs(vL);
        fR.s = o.sqrt(g * dR) + iabs(vR);
        double alpha = (SOLVER == LLF) ? imax(fL.s, fR.s) : 100.0;
        fL.h = 0.5 * ((vL * hL + vR * hR) + alpha * (QL.h - QR.h));
        fR.h = -fL.h;
        double sc = (vL * vL) * hL + (vR * vR) * hR;
        double pr = (0.5 * g) * (hL * hL + hR * hR);
        fL.p1 = 0.5 * ((sc + pr * n1) + alpha * (QL.p1 - QR.p1));
        fL.p2 = 0.5 * ((sc + pr * n2) + alpha * (QL.p2 - QR.p2));
        fR.p1 = -fL.p1;
        fR.p2 = -fL.p2;
    }
}

// The direction of a normal, as the fluxes take it: 1 = (+-1, +-0), 2 = (+-0, +-1), 0 = any other.
__device__ __forceinline__ int axis_of(double n1, double n2) {
    const long long one = 0x3ff0000000000000ll, a = abs_bits(n1), b = abs_bits(n2);
    return (a == one) & (b == 0) ? 1 : ((a == 0) & (b == one) ? 2 : 0);
}

// One edge: dL/dR are the depths h - b of the two states, sqL/sqR their
// sqrt(g * depth) and yL/yR recip_fix(depth) (only read for depths above the dry
// tolerance).
// With FastOps the updates count only where o.ok is true afterwards. SURFACE: see
// geoclaw_flux; the Lax-Friedrichs fluxes need the surface.
template <int SOLVER, int FZ, bool SURFACE = true, class Ops>
__device__ __forceinline__ void edge_flux(double n1, double n2, const State& QL, const State& QR, double dL,
                                          double dR, double sqL, double sqR, u64 yL, u64 yR, double drytol,
                                          Update& fL, Update& fR, int axis, uint16_t* fz, Ops& o) {
    if (SOLVER == FWAVE || SOLVER == AUG_RIEMANN)
        geoclaw_flux<SOLVER, FZ, SURFACE>(n1, n2, QL, QR, dL, dR, sqL, sqR, yL, yR, drytol, fL, fR, axis, fz, o);
    else
        lf_flux<SOLVER>(n1, n2, QL, QR, dL, dR, drytol, fL, fR, sqL, sqR, yL, yR, axis, o);
}

// depth, sqrt(g * depth) and recip_fix(depth) of a state, as the edge code needs them
__device__ __forceinline__ void depth_terms(const State& Q, double drytol, double& d, double& sq, u64& y) {
    d = Q.h - Q.b;
    const bool wet = lt(drytol, d);
    sq = wet ? sqrt_fix(kG * d) : 0.0;
    y = wet ? recip_fix(d) : 0;
}

// One edge between two states, for the entry points without a context, whose tolerance
// may be negative: a depth at or below zero is then wet. FastOps' quotients of zeros by
// a wet depth and the f-wave's shortcut for water at rest take that depth for positive,
// and the Lax-Friedrichs fluxes the root of a negative one for 0 (their
// sqrt(g max(d, 0))), the GeoClaw ones for NaN.
template <int SOLVER>
__device__ __forceinline__ void flux_of_states(double n1, double n2, const State& QL, const State& QR, double drytol,
                                               Update& fL, Update& fR) {
    double dL, dR, sqL, sqR;
    u64 yL, yR;
    depth_terms(QL, drytol, dL, sqL, yL);
    depth_terms(QR, drytol, dR, sqR, yR);
    if (SOLVER != FWAVE && SOLVER != AUG_RIEMANN) {
        if (lt0(dL)) sqL = 0.0;
        if (lt0(dR)) sqR = 0.0;
    }
    const int axis = axis_of(n1, n2);
    if (!lt0(drytol)) {
        FastOps f;
        edge_flux<SOLVER, 0>(n1, n2, QL, QR, dL, dR, sqL, sqR, yL, yR, drytol, fL, fR, axis, nullptr, f);
        if (f.ok) return;
    }
    SafeOps o;
    if ((SOLVER == FWAVE || SOLVER == AUG_RIEMANN) && lt0(drytol))
        geoclaw_rotated<SOLVER, 0>(n1, n2, QL, QR, dL, dR, sqL, sqR, yL, yR, drytol, fL, fR, axis, nullptr, o);
    else
        edge_flux<SOLVER, 0>(n1, n2, QL, QR, dL, dR, sqL, sqR, yL, yR, drytol, fL, fR, axis, nullptr, o);
}

// Ghost state of bnd_skeleton_scalar_op, src/SWE/SWE_euler_timestep.f90:231-255.
template <int BC>
__device__ __forceinline__ State boundary_ghost(double n1, double n2, const State& Q) {
    State g = Q;
    if (BC == BC_SLIP) {
        double d = z0(Q.p1 * n1) + Q.p2 * n2;
        g.p1 = Q.p1 - d * n1;
        g.p2 = Q.p2 - d * n2;
    } else if (BC == BC_NOSLIP) {
        g.p1 = -Q.p1;
        g.p2 = -Q.p2;
    }
    return g;
}

}  // namespace SWE_KNS
