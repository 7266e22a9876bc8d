// FP64 functions of near-pair integrals on the integer and FP32 pipes: sine and
// cosine, decaying exponential, square root and its reciprocal of a double,
// with the fixed-point primitives of the assembly.
//
// GB300 issues an FP64 instruction for a warp every 62 cycles per scheduler
// (measured), an IMAD.WIDE every 2.5: the library's sincos (some 35 FP64
// operations) and rsqrt (8) are most of a quadrature point's time.  Here the
// argument's bits are taken apart, the function is evaluated on 64-bit integers
// (about 150 and 80 instructions) and the double is put together from bits.
// Errors against extended precision: roots 0.51 ulp, exponential 0.7 ulp, sine
// and cosine 2^-59 of 1 besides the final rounding (an error of the modulus of
// e^{ikr}), the sine below 2^-8 0.51 ulp.  Arguments beyond the ranges below take
// the library's functions.  Measured: corrections of the near pairs of the mixed assembly at 11562
// nodes 232 -> 202 us and of the mixed product at 40962 nodes 1.56 -> 1.36 ms
// (which had sine and cosine in double-float), FP64 matrix-free product at 5762
// nodes 16.7 -> 11.7 ms.
//
// The host compiles this header too (the tests drive it on the CPU).
#pragma once

#include "bie_fix64.cuh"

#include <cstring>
#ifndef __CUDACC__
#include <cmath>
#endif

namespace bie {
namespace fix64 {

FX_FN u64 double_bits(double x) {
#ifdef __CUDA_ARCH__
    return (u64)__double_as_longlong(x);
#else
    u64 u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}
FX_FN double bits_double(u64 u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}
FX_FN int leading_zeros(u64 v) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return v ? __builtin_clzll(v) : 64;
#endif
}
FX_FN u64 mul_high(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}

// v 2^e as a double (round half up in magnitude); the result must be normal
FX_FN double fixed_double(i64 v, int e) {
    const u64 s = (u64)(v >> 63), a = ((u64)v ^ s) - s;
    const int z = leading_zeros(a);
    const u64 n = a << (z & 63);
    const u64 m = (n >> 11) + ((n >> 10) & 1);   // 53 bits and a carry
    const u64 bits = ((u64)(unsigned)(e + 1085 - z) << 52) + m;
    return a ? bits_double(bits | (s & ((u64)1 << 63))) : 0.0;
}

// rinv = 1 / sqrt(r2), r = sqrt(r2); false (nothing set) outside [2^-1000, 2^1000]
FX_FN bool root(double r2, double &rinv, double &r) {
    const u64 u = double_bits(r2);
    const int ex = (int)(u >> 52);
    if ((unsigned)(ex - 23) > 2000u) return false;
    const int h = (ex - 1023) >> 1, odd = (ex - 1023) & 1;
    const i64 m = (i64)(((u & 0xfffffffffffffull) | 0x10000000000000ull) << (6 + odd));   // r2 4^-h, Q58 in [1, 4)
    const Limb ml = split(m);
    const i64 ri = rcp_sqrt(m, ml);                        // Q61
    const Limb rl = split(ri);
    rinv = fixed_double(ri, -61 - h);
    r = fixed_double(fold_up<5>(wide(ml.h, rl.h), cross<5>(ml, rl) + hi32(wide(ml.l, rl.l))), -60 + h);
    return true;
}

// (m j + more) >> sh of a 53-bit and a 64-bit number, 0 < sh: the low 64 bits, the rest
// in top
FX_FN u64 scaled_product(u64 m, u64 j, int sh, u64 &top, u64 more = 0) {
    const u64 lo = m * j + more, hi = mul_high(m, j) + (lo < more ? 1 : 0);
    const int a = sh < 64 ? sh : 63, b = sh < 64 ? 0 : (sh < 127 ? sh - 64 : 63);
    top = sh < 64 ? hi >> a : 0;
    return sh < 64 ? (hi << (64 - a)) | (lo >> a) : hi >> b;
}

// sine of |x| < 2^-8 relative to x: x (1 - x^2 / 6 + x^4 / 120), to 2^-60 of x besides
// the final rounding.  u: the bits of x, ex: its biased exponent.
FX_FN double sine_small(double x, u64 u, int ex) {
    if (ex < 993) return x;                                            // |x| < 2^-30
    const u64 m = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << 11;   // |x| 2^(1086 - ex)
    const int sh = 2036 - 2 * ex;                                      // (8 .. 50)
    const u64 z = mul_high(m, m) >> sh;                                // x^2, Q72, < 2^56
    const u64 q = mul_high(z << 8, z << 8);                            // x^4, Q96
    const u64 p = mul_high(z, 3074457345618258603ull) - (mul_high(q, 153722867280912930ull) >> 24);   // Q72
    const u64 r = m - (mul_high(m, p) >> 8);
    const double s = fixed_double((i64)(r >> 1), ex - 1085);
    return (i64)u < 0 ? -s : s;
}

// sine and cosine of x; false (nothing set) from |x| >= 2^(kBeyond - 1023) on and for
// NaN, kBeyond at most 1076 (2^53)
template <int kBeyond = 1043, class Table>
FX_FN bool sine_cosine(double x, const Table &table, double &s, double &c) {
    const u64 u = double_bits(x);
    const int ex = (int)(u >> 52) & 0x7ff;
    if (ex >= kBeyond) return false;
    // x / 2 pi as a 64-bit fraction of a turn (a subnormal is below 2^-64): 2^66 / 2 pi
    // in two words, the second for |x| >= 2^9 (rounded to one word it is good to
    // 2^-69 |x|)
    const u64 m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    u64 top;
    const u64 frac = ex < 1032 ? scaled_product(m, 0xa2f9836e4e44152aull, 1077 - ex, top)
                               : scaled_product(m, 0xa2f9836e4e441529ull, 1077 - ex, top,
                                                mul_high(m, 0xfc2757d1f534ddc0ull));
    i64 Er, Ei;
    unit_circle<true>(frac, table, Er, Ei);
    c = fixed_double(Er, -62);
    // (small arguments: where e^{ikr} is nearly real its imaginary part is a result of
    // its own, and k r cos(k r) - sin(k r) cancels)
    s = ex < 1015 ? sine_small(x, u, ex) : fixed_double((i64)u < 0 ? -Ei : Ei, -62);
    return true;
}

// e^-x; false (nothing set) for |x| >= 700 and NaN
template <class Table>
FX_FN bool exp_minus(double x, const Table &table, double &v) {
    const u64 u = double_bits(x);
    const int ex = (int)(u >> 52) & 0x7ff;
    if ((u & 0x7fffffffffffffffull) >= 0x4085e00000000000ull) return false;
    // x log2(e) = top + frac 2^-64 (log2(e) 2^63)
    u64 top;
    u64 frac = scaled_product((u & 0xfffffffffffffull) | 0x10000000000000ull, 0xb8aa3b295c17f0bcull, 1074 - ex, top);
    if ((i64)u < 0) {
        frac = (u64)0 - frac;
        top = ~top + (frac == 0 ? 1 : 0);
    }
    int carry;
    const i64 w = exp2_fraction(frac, carry, table);
    v = fixed_double(w, -62 - (int)(i64)top - carry);
    return true;
}

// ---- IEEE division and square root, rounded to nearest even ----------------
// From an approximation of the quotient (root) to 2^-60 and the exact remainder
// in 64-bit arithmetic, so the double is the one of the FP64 pipe's sequence.

// 1 / B in Q62 of (1, 2], B: Q64 in [1/2, 1), to a few units: a float estimate and
// two Newton steps
FX_FN u64 reciprocal(u64 B) {
    const float b = u32_to_float((unsigned)(B >> 32)) * 0x1p-32f;
    const u64 y0 = (u64)(unsigned)round_to_int((1.0f / b) * 0x1p29f) << 33;      // Q62, 2^-23
    const i64 e1 = (i64)(((u64)1 << 62) - mul_high(B, y0));                      // 1 - b y0, Q62
    const u64 y1 = y0 + (u64)(wide((int)(e1 >> 10), (int)(y0 >> 33)) >> 19);     // Q62, 2^-45
    const i64 e2 = (i64)(((u64)1 << 62) - mul_high(B, y1));
    return y1 + (u64)(wide((int)e2, (int)(y1 >> 33)) >> 29);
}
FX_FN u64 mantissa(double x) { return (double_bits(x) & 0xfffffffffffffull) | 0x10000000000000ull; }
FX_FN int exponent(double x) { return (int)(double_bits(x) >> 52) & 0x7ff; }

// Division by one positive normal b
struct Divisor {
    u64 mb, R;
    int eb;
};
FX_FN Divisor divisor(double b) {
    const u64 mb = mantissa(b);
    return Divisor{mb, reciprocal(mb << 11), exponent(b)};
}
// a / b for a zero or normal a and a normal quotient
FX_FN double divide(double a, const Divisor &d) {
    const u64 ma = mantissa(a);
    const int s = ma < d.mb ? 1 : 0;
    // ma 2^(53 + s) / mb in [2^53, 2^54); the reciprocal is of mb 2^-53
    u64 Q = mul_high(ma << (9 + s), d.R) >> 7;
    i64 rem = (i64)((ma << (53 + s)) - Q * d.mb);          // (the true value is small)
    if (rem < 0) { --Q; rem += (i64)d.mb; }
    if (rem >= (i64)d.mb) { ++Q; rem -= (i64)d.mb; }
    const u64 m = (Q >> 1) + (Q & 1 & ((rem != 0 ? 1 : 0) | (Q >> 1)));
    const u64 bits = ((u64)(unsigned)(exponent(a) - d.eb + 1022 - s) << 52) + m;
    const u64 sign = double_bits(a) & ((u64)1 << 63);
    return bits_double(exponent(a) == 0 ? sign : (bits | sign));
}
// sqrt of x in [1, 4)
FX_FN double square_root(double x) {
    const u64 mx = mantissa(x) << (exponent(x) - 1023);    // x in Q52
    const i64 q = (i64)(mx << 6);                          // Q58
    const Limb l = split(q), ri = split(rcp_sqrt(q, l));
    u64 T = (u64)fold_up<5>(wide(l.h, ri.h), cross<5>(l, ri) + hi32(wide(l.l, ri.l))) >> 7;   // Q53
    i64 rem = (i64)((mx << 54) - T * T);
    if (rem < 0) { --T; rem += (i64)(2 * T + 1); }
    if (rem > (i64)(2 * T)) ++T;
    return bits_double(((u64)1022 << 52) + (T >> 1) + (T & 1));
}
// Julia's 3-argument hypot (maximum-abs scaling, IEEE division and square root,
// ((a^2 + b^2) + c^2) summation), bit for bit; false (nothing set) where a
// component other than zero is below 2^-100 times the largest, or that one
// outside [2^-900, 2^900]
FX_FN double mul_rn(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
FX_FN double add_rn(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
FX_FN double magnitude(double x) { return bits_double(double_bits(x) & 0x7fffffffffffffffull); }
FX_FN bool hypot3(double x, double y, double z, double &h) {
    const u64 ux = double_bits(magnitude(x)), uy = double_bits(magnitude(y)), uz = double_bits(magnitude(z));
    u64 um = ux > uy ? ux : uy;
    um = uz > um ? uz : um;
    const double m = bits_double(um);
    const int em = exponent(m);
    if ((unsigned)(em - 123) > 1800u) return false;
    const u64 low = um - ((u64)100 << 52);                 // 2^-100 m
    if ((ux != 0 && ux < low) || (uy != 0 && uy < low) || (uz != 0 && uz < low)) return false;
    const Divisor d = divisor(m);
    const double a = divide(x, d), b = divide(y, d), c = divide(z, d);
    h = mul_rn(m, square_root(add_rn(add_rn(mul_rn(a, a), mul_rn(b, b)), mul_rn(c, c))));
    return true;
}

}  // namespace fix64

#ifdef __CUDACC__
namespace dev {

// out of line: the ranges of no quadrature point of a sound mesh
static __device__ __noinline__ double2 sincos_library(double x) {
    double s, c;
    sincos(x, &s, &c);
    return make_double2(s, c);
}
static __device__ __noinline__ double exp_library(double x) { return exp(x); }

// The functions above as element_fp64 takes them; tab: the context's tables of
// e^{2 pi i j / 1024} and 2^(-j / 256) as limbs.
struct TrigFix {
    const int32_t *tab;
    __device__ __forceinline__ void sincos_of(double x, double *s, double *c) const {
        auto table = [&](int j, fix64::Limb &tc, fix64::Limb &ts) {
            const int4 t = __ldg(reinterpret_cast<const int4 *>(tab) + j);
            tc = fix64::Limb{t.x, t.y};
            ts = fix64::Limb{t.z, t.w};
        };
        // (far field points, whose every pair may come here: with the library from
        // 2^20 on 30000 points at k r = 10^8 took 113 ms, the FP64 kernel 96)
        if (fix64::sine_cosine<1076>(x, table, *s, *c)) return;
        const double2 v = sincos_library(x);
        *s = v.x;
        *c = v.y;
    }
    __device__ __forceinline__ void root_of(double r2, double &rinv, double &r) const {
        if (fix64::root(r2, rinv, r)) return;
        rinv = rsqrt(r2);
        r = r2 * rinv;
    }
    __device__ __forceinline__ double exp_minus(double x) const {
        auto table = [&](int j) {
            const int2 t = __ldg(reinterpret_cast<const int2 *>(tab + 4 * fix64::kTrigEntries) + j);
            return fix64::Limb{t.x, t.y};
        };
        double v;
        return fix64::exp_minus(x, table, v) ? v : exp_library(-x);
    }
};

}  // namespace dev
#endif
}  // namespace bie
