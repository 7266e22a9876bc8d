// 64-bit fixed-point evaluation of one regular (target, element) pair at FP64
// accuracy on the integer and FP32 pipes.
//
// GB300 issues FP64 instructions at 1/64 of the FP32 rate (2 against 128 lanes
// per clock and SM, measured), while a 32 x 32 + 64 bit multiply-add
// (IMAD.WIDE) runs at 64.  A regular pair has known magnitudes (its points are
// at least half the centroid's distance away), so every value of the
// quadrature sequence can be carried as a 64-bit integer with a scale the pair
// fixes once: a product costs three or four IMAD.WIDE where the FP64 pipe
// would take 64 issue slots, and sums are exact.  The scales below keep the
// rounding of each step at 2^-54 .. 2^-60 of the value's range, at or below an
// FP64 rounding.
//
// Notation: "Qn" is an integer v standing for v 2^-n.  A limb pair {h, l}
// stands for h 2^32 + l with a signed low limb, so that every partial product
// is a signed 32 x 32 multiply and sums of products need no carries.
//
// Pair normalisation: lengths in units of 2^e with rmin = |D| - rho in
// [1/2, 1) 2^e (D = centroid - target, rho = largest point or node offset of
// the element); regular pairs have |D| >= 2.01 rho, so r lies in [1/2, 3) and
// 1/r in (1/3, 2].
//
// The host compiles this header too (the tests drive the same functions
// against extended precision on the CPU).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define FX_FN __host__ __device__ __forceinline__
#else
#define FX_FN inline
#include <cmath>
#endif

namespace bie {
namespace fix64 {

typedef long long i64;
typedef unsigned long long u64;

struct Limb {
    int h, l;
};

// a b and acc + a b, signed 32 x 32 -> 64 (left to itself the compiler widens
// some operands first and multiplies 64 x 64)
FX_FN i64 wide(int a, int b) {
#ifdef __CUDA_ARCH__
    i64 r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r;
#else
    return (i64)a * (i64)b;
#endif
}
FX_FN i64 wide_add(i64 acc, int a, int b) {
#ifdef __CUDA_ARCH__
    i64 r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(acc));
    return r;
#else
    return acc + (i64)a * (i64)b;
#endif
}
FX_FN int hi32(i64 x) { return (int)(x >> 32); }
FX_FN int lo32(i64 x) { return (int)(unsigned)(u64)x; }
FX_FN i64 make64(int h, unsigned l) { return (i64)(((u64)(unsigned)h << 32) | (u64)l); }
// x >> n for n >= 0 (everything but the sign from 63 on)
FX_FN i64 shift_right(i64 x, int n) {
#ifdef __CUDA_ARCH__
    i64 r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
    return r;
#else
    return x >> (n < 63 ? n : 63);
#endif
}
// H + (L >> 32)
FX_FN i64 fold(i64 H, i64 L) { return wide_add(H, hi32(L), 1); }
// h 2^32 + l with l signed; |x| < 2^63 - 2^31
FX_FN Limb split(i64 x) { return Limb{(int)((unsigned)hi32(x) + ((unsigned)lo32(x) >> 31)), lo32(x)}; }
// acc + a.h b.h, and the cross products acc + a.h b.l + a.l b.h
FX_FN i64 high(i64 acc, Limb a, Limb b) { return wide_add(acc, a.h, b.h); }
FX_FN i64 cross(i64 acc, Limb a, Limb b) { return wide_add(wide_add(acc, a.h, b.l), a.l, b.h); }
// ... from one half, so that the shift in fold() / fold_up<S>() rounds: sums of
// many terms (the C row sums cancel) would see the bias of a truncation
template <int S = 0>
FX_FN i64 cross(Limb a, Limb b) {
    return cross((i64)1 << (31 - S), a, b);
}
// a b 2^-64, rounded (the product of the low limbs is left out)
FX_FN i64 mulhi(Limb a, Limb b) { return fold(wide(a.h, b.h), cross(a, b)); }
// (H 2^32 + L) >> (32 - S), 0 < S < 32
template <int S>
FX_FN i64 fold_up(i64 H, i64 L) { return (i64)((u64)H << S) + (L >> (32 - S)); }
// (a b) >> (64 - S)
template <int S>
FX_FN i64 mulhi_up(Limb a, Limb b) { return fold_up<S>(wide(a.h, b.h), cross<S>(a, b)); }

// (ar + i ai) (br + i bi) 2^-62, b in Q62
struct Values2 {
    i64 re, im;
};
FX_FN Values2 complex_mul(Limb ar, Limb ai, Limb br, Limb bi) {
    const Limb mbi = split(-((i64)((u64)(i64)bi.h << 32) + (i64)bi.l));
    return Values2{fold_up<2>(high(wide(ar.h, br.h), ai, mbi), cross(cross<2>(ar, br), ai, mbi)),
                   fold_up<2>(high(wide(ar.h, bi.h), ai, br), cross(cross<2>(ar, bi), ai, br))};
}

// An element's complex factor on G as Q62 limbs times 2^-e and that e, its own
// exponent (largest component in [1/2, 1)): factors of a mesh may spread over any
// range without losing bits.  Zero has the exponent kZeroFactor, below every
// other one's.
constexpr int kZeroFactor = -4096;
struct Factor {
    Limb re, im;
    int e;
};
FX_FN Factor element_factor(double re, double im) {
    const double m = re < 0 ? -re : re, n = im < 0 ? -im : im, top = m > n ? m : n;
    if (top == 0.0) return Factor{Limb{0, 0}, Limb{0, 0}, kZeroFactor};
#ifdef __CUDA_ARCH__
    int e;
    (void)frexp(top, &e);
    return Factor{split(__double2ll_rn(ldexp(re, 62 - e))), split(__double2ll_rn(ldexp(im, 62 - e))), e};
#else
    int e;
    (void)std::frexp(top, &e);
    return Factor{split((i64)std::llrint(std::ldexp(re, 62 - e))), split((i64)std::llrint(std::ldexp(im, 62 - e))), e};
#endif
}

constexpr int kTrigBits = 10;                      // e^{2 pi i j / 1024}
constexpr int kTrigEntries = 1 << kTrigBits;
constexpr int kCoordBits = 59;                     // fixed coordinates: largest |x| -> 2^59
constexpr int kMinExp = -7;                        // pairs with rmin < 2^(kMinExp - 1) go to FP64
constexpr float kRhoFactor = 2.01f;                // regular: |D| >= kRhoFactor rho
constexpr int kMaxTurnExp = 25;                    // k 2^e / 2 pi < 2^25 (Pair::fsh below 32)
constexpr int kDampBits = 8;                       // 2^(-j / 256)
constexpr int kDampEntries = 1 << kDampBits;
constexpr int kMaxDampExp = 9;                     // |Im k| 2^e log2(e) < 2^9
constexpr float kMaxDampSpread = 1.5f;             // |Im k| rho log2(e) of a regular pair

// 2 pi / 1024 in Q65 (2 pi 2^55 rounded)
constexpr i64 kStepQ65 = 226375608064910089LL;

// What a pair fixes for its quadrature points.
struct Pair {
    i64 Dx, Dy, Dz;      // centroid - target, Q61 of 2^e
    int osh;             // right shift of the point offsets
    Limb Km;             // k 2^e / 2 pi 2^-ks, Q62
    int fsh;             // 6 + ks: turns of P (Q58) to 64 fraction bits
    Limb kq;             // Re k 2^(e - fe), Q61
    int fe;              // F and k r t are carried times 2^-fe
    // complex k: e^{-Im k r} = 2^-x, x = Im k r log2(e), carried times 2^base
    Limb Kd;             // Im k 2^e log2(e) 2^-ds, Q62
    int dsh;             // 6 + ds
    int base;            // at most floor(x) over the element
    Limb kiq;            // Im k 2^(e - fe), Q61
};

// Values of one quadrature point.
struct Point {
    i64 Fr, Fi, Gr, Gi;  // Q58: F in 2^(ej - 2e + fe), G in 2^(ej - e)
    i64 tq;              // Q57: t in 2^(ej - 2e), C_q = -t
};

// Point data as stored in the record (16 words): offsets from the centroid
// Q62 of 2^eo, unit normal Q61 limbs, jw / 4 pi Q63 of 2^ej limbs.
struct PointData {
    i64 ox, oy, oz;
    Limb nx, ny, nz, jw;
};

// 1 / sqrt of a float: the start value of the reciprocal's correction
FX_FN float rsqrt_start(float x) {
#ifdef __CUDA_ARCH__
    return rsqrtf(x);
#else
    return 1.0f / std::sqrt(x);
#endif
}
FX_FN float std_abs(float x) { return x < 0.0f ? -x : x; }
FX_FN float u32_to_float(unsigned u) { return (float)u; }
FX_FN int round_to_int(float x) {
#ifdef __CUDA_ARCH__
    return __float2int_rn(x);
#else
    return (int)std::nearbyint(x);
#endif
}

// 1 / r in Q61 from r^2 in Q58 (r in [1/2, 3)): float estimate and one
// third-order correction y0 (1 + c/2 + 3 c^2 / 8), c = 1 - r^2 y0^2
FX_FN i64 rcp_sqrt(i64 r2, Limb r2l) {
    const unsigned u = (unsigned)(u64)(r2 >> 30);                      // Q28
    const int y0 = round_to_int(rsqrt_start(u32_to_float(u)) * 4398046511104.0f);   // Q28 (times 2^42)
    const Limb t = split(wide(y0, y0));                                // Q56
    const i64 H = wide(r2l.h, t.h);                                    // 2^64 units of Q114
    const i64 L = fold(cross(0, r2l, t), wide(r2l.l, t.l));
    const i64 e = -(i64)(((u64)(H - ((i64)1 << 50)) << 32) + (u64)L);  // Q82
    const i64 e2 = wide(hi32(e), hi32(e));                             // Q100
    const i64 c = wide_add(e, hi32(e2), 12288);                        // Q83: e/2 + 3 e^2/8
    const Limb cl = split(c);
    const i64 W = fold(wide(y0, cl.h), wide(y0, cl.l));                // Q79
    return (i64)((u64)(i64)y0 << 33) + (W >> 18);
}

// E = e^{i theta} (Q62) from theta as a 64-bit fraction of a turn: the table
// entry T nearest below or above plus T (cos d - 1 + i sin d), |d| <= pi / 1024.
// Largest error 2^-55 (the series in 32-bit steps), FINE 2^-60.
template <bool FINE = false, class Table>
FX_FN void unit_circle(u64 frac, const Table &table, i64 &Er, i64 &Ei) {
    const unsigned top = (unsigned)(frac >> 32) + 0x00200000u;
    Limb Tc, Ts;
    table((int)(top >> 22), Tc, Ts);
    // remainder in (-1/2, 1/2] table steps, Q63
    const unsigned rh = (unsigned)(frac >> 32) - (top & 0xffc00000u);
    const i64 f = (i64)((((u64)rh << 32) | (u64)(unsigned)frac) << 9);
    const Limb C = split(kStepQ65);
    const i64 d = mulhi(split(f), C);                                  // angle, Q64, |d| < 2^55.7
    const Limb dl = split(d);
    const i64 z = wide_add(wide(dl.h, dl.h), hi32(wide(dl.h, dl.l)), 2);   // d^2, Q64
    const int zA = (int)(z >> 17);                                     // Q47
    const i64 z3 = wide(zA, 1431655765);                               // d^2 / 3, Q79
    const int q = hi32(wide(zA, hi32(z3)));                            // d^4 / 3, Q62
    i64 sn, c1 = ((i64)q - z) >> 1;                                    // sin and cos - 1, Q64
    if (FINE) {
        // d^2/6 - d^4/120 in Q77, and the next term of cos
        const i64 w = mulhi(split((i64)((u64)z << 13)), split(3074457345618258603LL)) - (wide(q, 26214) >> 5);
        sn = d - ((mulhi(dl, split(w)) + 4096) >> 13);
        c1 -= (i64)hi32(wide(hi32(wide(q, zA)), 2185));
    } else {
        const int w = hi32(wide_add(z3, q, -6554));                    // d^2/6 - d^4/120, Q48
        const int dA = (int)(d >> 25);                                 // Q39
        const int dw = (int)(wide(dA, w) >> 29);                       // Q58
        sn = wide_add(d, dw, -64);
    }
    const Limb s = split(sn), ms = split(-sn);
    const Limb c = split(c1);
    Er = fold(make64(Tc.h, 0) + (i64)Tc.l + high(wide(Tc.h, c.h), Ts, ms), cross(cross(Tc, c), Ts, ms));
    Ei = fold(make64(Ts.h, 0) + (i64)Ts.l + high(wide(Ts.h, c.h), Tc, s), cross(cross(Ts, c), Tc, s));
}

// 2^-(f - carry) (Q62), f = frac 2^-64: the next table entry below or above
// (carry) times a series
template <class Table>
FX_FN i64 exp2_fraction(u64 frac, int &carry, const Table &table) {
    const u64 up = frac + ((u64)1 << 55);
    carry = up < frac ? 1 : 0;
    const Limb Td = table((int)(up >> 56));
    const i64 f = (i64)((frac - (up & 0xff00000000000000ull)) << 7);  // Q63 of a table step
    const Limb C = split(99893036290645747LL);                        // ln 2 / 256, Q65
    const i64 u = mulhi(split(f), C);                                  // Q64, |u| < 2^-9.5
    const Limb ul = split(u);
    const i64 u2 = wide_add(wide(ul.h, ul.h), hi32(wide(ul.h, ul.l)), 2);   // Q64
    const int uA = (int)(u >> 24), u2A = (int)(u2 >> 15);              // Q40, Q49
    const int u3 = hi32(wide(uA, u2A));                                // Q57
    const int u4 = hi32(wide(u2A, u2A));                               // Q66
    const int u5 = hi32(wide(uA, u4));                                 // Q74
    // e^-u - 1 = -u + u^2/2 - u^3/6 + u^4/24 - u^5/120
    i64 p = (u2 >> 1) - u;
    p = wide_add(p, hi32(wide(u3, 715827883)), -128);
    p += (i64)hi32(wide(u4, 44739243)) - (i64)hi32(wide(u5, 34953));
    return make64(Td.h, 0) + (i64)Td.l + mulhi(Td, split(p));
}

// 2^-(x - base) (Q62) from x = T 2^(6 + ds) 2^-64 (T: Q58 of 2^ds, tl: the next 32
// bits) and the table of 2^(-j / 256) limbs
template <class Table>
FX_FN i64 damping(i64 T, unsigned tl, int dsh, int base, const Table &table) {
    const u64 frac = ((u64)T << dsh) | (u64)(tl >> (32 - dsh));
    int carry;
    const i64 v = exp2_fraction(frac, carry, table);
    return shift_right(v, (int)(T >> (64 - dsh)) + carry - base);
}

// One quadrature point of a regular pair: greens3d!, freens3d!, freens3dk0!
// (src/3d/kernels.jl:13-55) times the jacobian-weight product
// (src/3d/assembly_collocation.jl:213-252).
template <bool CPLX_K, class Table, class DampTable>
FX_FN Point point(const PointData &g, const Pair &P, const Table &table, const DampTable &damp_table) {
    const i64 dx = P.Dx + (g.ox >> P.osh), dy = P.Dy + (g.oy >> P.osh), dz = P.Dz + (g.oz >> P.osh);   // Q61
    const Limb x = split(dx), y = split(dy), z = split(dz);
    i64 H = wide_add(wide_add(wide(x.h, x.h), y.h, y.h), z.h, z.h);
    i64 L = wide_add(wide_add(wide(x.h, x.l), y.h, y.l), z.h, z.l);
    const i64 r2 = wide_add(H, hi32(L), 2);                            // Q58
    const Limb r2l = split(r2);
    const Limb ri = split(rcp_sqrt(r2, r2l));                          // 1/r, Q61
    // phase: r (Q60) times k/2pi, its fraction of a turn
    const Limb r = split(mulhi_up<5>(r2l, ri));
    L = cross(0, r, P.Km);
    const i64 T = fold(wide(r.h, P.Km.h), L);                          // Q58 of 2^ks, 32 more bits in L
    const u64 frac = ((u64)T << P.fsh) | (u64)((unsigned)lo32(L) >> (32 - P.fsh));
    i64 Er, Ei;
    unit_circle(frac, table, Er, Ei);
    if (CPLX_K) {
        L = cross(0, r, P.Kd);
        const i64 x = fold(wide(r.h, P.Kd.h), L);
        const Limb dm = split(damping(x, (unsigned)lo32(L), P.dsh, P.base, damp_table));
        Er = mulhi_up<2>(split(Er), dm);
        Ei = mulhi_up<2>(split(Ei), dm);
    }
    const Limb er = split(Er), ei = split(Ei), mei = split(-Ei);
    // (x - y).n and the cosine of its angle
    H = high(high(wide(x.h, g.nx.h), y, g.ny), z, g.nz);
    L = cross(cross(cross(x, g.nx), y, g.ny), z, g.nz);
    const Limb dn = split(fold(H, L));                                 // Q58
    const Limb cs = split(mulhi_up<7>(dn, ri));                        // Q62
    const Limb wg = split(mulhi(ri, g.jw));                            // jw / 4 pi r, Q60
    Point v;
    v.Gr = mulhi(er, wg);
    v.Gi = mulhi(ei, wg);
    const Limb m1 = split(mulhi(cs, wg));                              // Q58
    H = wide(m1.h, ri.h);
    const i64 t = fold_up<5>(wide(m1.h, ri.h), cross(0, m1, ri));      // Q60
    v.tq = (t + 4) >> 3;                                               // Q57, rounded: C sums cancel
    i64 mt_ = -(t >> P.fe);                                            // -t 2^-fe, Q60
    if (CPLX_K) mt_ -= mulhi_up<5>(m1, P.kiq);                         // -(1 + Im k r) t 2^-fe
    const Limb mt = split(mt_);
    const Limb tk = split(mulhi_up<5>(m1, P.kq));                      // k r t 2^-fe, Q60
    // F = e^{ikr} (i k r - 1) t
    v.Fr = fold(high(wide(er.h, mt.h), mei, tk), cross(cross(er, mt), mei, tk));
    v.Fi = fold(high(wide(er.h, tk.h), ei, mt), cross(cross(er, tk), ei, mt));
    return v;
}

// Exponent x with v in [2^(x-1), 2^x) for a positive normal float
FX_FN int float_exp(float v) {
#ifdef __CUDA_ARCH__
    return ((__float_as_int(v) >> 23) & 255) - 126;
#else
    int x;
    std::frexp(v, &x);
    return x;
#endif
}

// k 2^e as the pair's phase and amplitude factors.  km, kx: Re k / 2 pi = km
// 2^-62 2^kx with |km| in [2^61, 2^62) (or 0); ka, kb: Re k = ka 2^-62 2^kb
// with |ka| < 2^62.
FX_FN void pair_wavenumber(Pair &P, i64 km, int kx, i64 ka, int kb, int e) {
    const int a = kx + e, ks = a > 0 ? a : 0, sh = a < 0 ? (-a < 63 ? -a : 63) : 0;
    P.Km = split(km >> sh);
    P.fsh = 6 + ks;
    const int b = kb + e;
    P.fe = b > 1 ? b - 1 : 0;
    const int s = 1 - (b - P.fe);                // Q61 of a value below 2
    P.kq = split(ka >> (s < 63 ? s : 63));
}
// The same for Im k: kd, kdx: Im k log2(e) = kd 2^-62 2^kdx; kai: Im k = kai 2^-62
// 2^kb with the exponent of Re k (|kai|, |ka| < 2^61).  base: pair_base.
FX_FN void pair_damping(Pair &P, i64 kd, int kdx, i64 kai, int kb, int e, int base) {
    const int a = kdx + e, ds = a > 0 ? a : 0, sh = a < 0 ? (-a < 63 ? -a : 63) : 0;
    P.Kd = split(kd >> sh);
    P.dsh = 6 + ds;
    P.base = base;
    const int s = 1 - (kb + e - P.fe);
    P.kiq = split(kai >> (s < 63 ? s : 63));
}
FX_FN int floor_to_int(float x) {
#ifdef __CUDA_ARCH__
    return __float2int_rd(x);
#else
    return (int)std::floor(x);
#endif
}
// x of a point is at least kl r0 - |kl| rho (kl = Im k log2(e), r0 = |D|), less a
// margin for FP32
FX_FN int pair_base(float kl, float r0, float rho) {
    return floor_to_int(kl * r0 - std_abs(kl) * rho * 1.0001f - 0.01f);
}
// base of an entry at distance d: at most the base of every pair that adds to it
// (its node is within rho of the pair's centroid)
FX_FN int entry_base(float kl, float d, float rho_max) {
    return floor_to_int(kl * d - 2.0f * std_abs(kl) * rho_max * 1.0001f - 0.02f) - 1;
}
// |F| of the element's entries is carried times 2^-fe (see pair_wavenumber)
FX_FN int amplitude_exp(int kb, int e) { return kb + e > 1 ? kb + e - 1 : 0; }

// Scales of an entry (row, node): all its contributions are summed as 64-bit
// integers in units of 2^(entry exponent), a function of the row-node distance
// alone (fl = floor(log2 distance), computed the same way by every element that
// touches the node) and of the node's largest element weight exponent ej.  A
// pair has e >= fl - 1 (r_min >= distance / 3), so its own unit
// 2^(ej_e - e - 55) [G], 2^(ej_e - 2e + fe - 55) [F] is never coarser.
FX_FN int entry_exp_g(int ej, int fl) { return ej - (fl - 1) - 55; }
FX_FN int entry_exp_f(int ej, int fl, int kb) { return ej - 2 * (fl - 1) + amplitude_exp(kb, fl - 1) - 55; }

// Byte offset of a node's column of complex128 entries, rows in a column
FX_FN u64 column_bytes(int node, i64 rows) { return (u64)(unsigned)node * (u64)rows << 4; }

// Place in the list of deferred pairs of pair pe of a (row, slice), whose pairs come
// in order: true and its slot, or false where the list is full.  Such a row's
// slice is gone through again from over_at, its first pair without a place, so
// later pairs need none and do not count: the counter ends at most one above the
// list's length for each (row, slice), whatever the number of deferred pairs.
constexpr int kNoOverflow = 0x7fffffff;
template <class Count>
FX_FN bool defer_slot(Count count, u64 capacity, int pe, int &over_at, u64 &slot) {
    if (over_at < pe) return false;
    slot = count();
    if (slot < capacity) return true;
    over_at = pe;
    return false;
}

}  // namespace fix64
}  // namespace bie
