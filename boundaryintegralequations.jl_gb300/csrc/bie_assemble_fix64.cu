// K10: FP64-grade dense collocation assembly on the integer pipes
// (BIE_PREC_FP64 and BIE_PREC_DF64, real and complex k).
//
// Same result as K1 (assemble_parallel!, src/3d/assembly_collocation.jl:
// 270-479).  K1 is bound by the FP64 pipe, which GB300 runs at 1/64 of its
// FP32 rate (86 % busy); here the regular pairs are evaluated in 64-bit fixed
// point (bie_fix64.cuh), whose error is at or below FP64 rounding, and only the
// near pairs and nearest-node near-ties stay in FP64 (a list and a correction
// kernel, as in the mixed assembly).
//
// Measured (GB300, complete step): pulsating sphere, 10242 nodes, 3-node
// physics 133.3 -> 20.8 ms; 362 nodes, 16-point rules 0.79 -> 0.23 ms;
// BIE_PREC_DF64 (before: double-float kernel) 5762 nodes, 6-node physics
// 4.98 -> 3.24 ms, 11562 nodes 17.3 -> 11.3 ms.  Errors against a 64-bit
// evaluation are unchanged (pulsating sphere F 7.6e-14, dominated by near
// pairs).
// What bounds it now: instruction issue.  One point costs about 268
// instructions (71 IMAD.WIDE) = 528 issue cycles per warp, a node's output
// about 130 (48 IMAD.WIDE); measured per warp instruction IMAD.WIDE takes 2.45
// cycles, shifts and logic 2.1, adds 1.2 and they do not overlap.  Not kept:
// staging records in shared memory (same time as reading them through L1, plus
// barriers), 3 or 5 resident blocks (+5 %), all four points of a group at once
// (+15 %), integer-to-double conversion without the FP64 pipe (+3 %).
//
//   * one thread per target row, element slices in grid.y, records read through
//     L1 (every lane of a warp reads the same words);
//   * per pair the FP32 nearest-node choice with a near-tie margin, D = c - t as
//     integers, and the scales of the pair;
//   * per point the kernel values as integers, two points side by side; the
//     values of four points go through shared memory to the sums with the
//     physics basis (three IMAD.WIDE each: high x high and the two cross
//     products), so that neither loop holds the other's registers (128 against
//     214, 4 blocks per SM instead of 2: 4.4 -> 3.3 ms at 5762 nodes);
//   * each (row, node) entry is a running 64-bit integer sum in units fixed by
//     the row-node distance and the node's element weights, so sums are exact
//     and independent of their order: the first contribution in the node's
//     slice stores, later ones add, the last one converts to complex128; nodes
//     shared between slices take 64-bit integer atomics and a widening pass.
#include "bie_internal.h"
#include "bie_device.cuh"
#include "bie_fixmath.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

namespace bie {

namespace {

using dev::RuleInfo;
using fix64::i64;
using fix64::Limb;
using fix64::u64;
constexpr int kThreads = 128;
constexpr int kPointWords = 16;

// header words of a record
constexpr int kHdrNear2 = 0, kHdrRho = 1, kHdrEj = 2, kHdrEo = 3, kHdrCen = 4, kHdrNodes = 12;

struct Fp64View {
    const double *rec;
    int stride;
    int nidx_off;
    const double *phi;   // global, R x qmax x NP
    int qmax;
    RuleInfo ri;
    const int32_t *tab;   // tables of dev::TrigFix
};

// Scales of a launch (host values)
struct FxScale {
    double x0[3];        // origin of the scaled coordinates
    double inv;          // 2^-S
    double len;          // 2^S
    int S;
    int pe;              // basis values are stored times 2^-pe
    int extra;           // entry units times 2^extra (large node valences)
    float rho_max;       // largest rho of the mesh
    int extra_w;         // the same for G with element factors
};

// k as mantissas and exponents (see fix64::pair_wavenumber, pair_damping)
struct FxWave {
    i64 km, ka;          // Re k / 2 pi, Re k
    i64 kd, kai;         // Im k log2(e), Im k
    int kx, kb, kdx;
    float kl;            // Im k log2(e)
    float rho_max;       // largest rho of the mesh
};

// integer nearest to (hi + lo) 2^n, |hi| 2^n below 2^62
__device__ __forceinline__ i64 fx_round(double hi, double lo, int n) {
    return __double2ll_rn(ldexp(hi, n)) + __double2ll_rn(ldexp(lo, n));
}

template <bool CPLX_K>
__device__ __forceinline__ FxWave fx_wave(double kre, double kim, const FxScale &sc) {
    // 1 / 2 pi and log2(e) as hi + lo
    constexpr double kHi = 0x1.45f306dc9c883p-3, kLo = -0x1.6b01ec5417056p-57;
    constexpr double lHi = 0x1.71547652b82fep+0, lLo = 0x1.777d0ffda0d24p-56;
    const double k = kre * sc.len, ki = kim * sc.len;
    FxWave w{0, 0, 0, 0, -1000, -1000, -1000, 0.f, sc.rho_max};
    if (k != 0.0) {
        const double hi = k * kHi, lo = fma(k, kHi, -hi) + k * kLo;
        (void)frexp(hi, &w.kx);
        (void)frexp(k, &w.kb);
        w.km = fx_round(hi, lo, 62 - w.kx);
    }
    if (CPLX_K) {
        int kb2 = -1000;
        if (ki != 0.0) {
            const double hi = ki * lHi, lo = fma(ki, lHi, -hi) + ki * lLo;
            (void)frexp(hi, &w.kdx);
            (void)frexp(ki, &kb2);
            w.kd = fx_round(hi, lo, 62 - w.kdx);
            w.kl = (float)hi;
        }
        w.kb = max(w.kb, kb2) + 1;   // |Re k|, |Im k| below 2^(kb - 1)
        if (ki != 0.0) w.kai = fx_round(ki, 0.0, 62 - w.kb);
    }
    if (k != 0.0) w.ka = fx_round(k, 0.0, 62 - w.kb);
    return w;
}

// Units of an entry (row, node): floor(log2 |t - x|) of the FP32 coordinates and,
// for complex k, the base of its damping; evaluated the same way wherever they
// are needed
struct FxEntry {
    int fl, base;
};
template <bool CPLX_K>
__device__ __forceinline__ FxEntry fx_entry(float tx, float ty, float tz, float x, float y, float z, const FxWave &w) {
    const float dx = __fsub_rn(x, tx), dy = __fsub_rn(y, ty), dz = __fsub_rn(z, tz);
    const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
    return FxEntry{(fix64::float_exp(d2) - 1) >> 1, CPLX_K ? fix64::entry_base(w.kl, __fsqrt_rn(d2), w.rho_max) : 0};
}

// integer sum in units of 2^e as a double
template <bool CPLX_K>
__device__ __forceinline__ double fx_double(i64 v, int e) {
    const double d = (double)v;
    if (CPLX_K) return ldexp(d, e);   // strong damping may leave the normal range
    // real k: exponents stay far inside it (coordinates within 2^+-300)
    return v == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (e << 20), __double2loint(d));
}
template <bool CPLX_K>
__device__ __forceinline__ longlong2 fx_complex(longlong2 v, int e) {
    return make_longlong2(__double_as_longlong(fx_double<CPLX_K>(v.x, e)),
                          __double_as_longlong(fx_double<CPLX_K>(v.y, e)));
}

struct FxTarget {
    i64 x, y, z;         // fixed coordinates, 2^(59 - st) units
    float fx, fy, fz;    // scaled FP32 coordinates
    int st;
    bool bad;            // not representable: every pair in FP64
};

__device__ __forceinline__ FxTarget fx_target(double tx, double ty, double tz, const FxScale &sc) {
    FxTarget T;
    const double x = (tx - sc.x0[0]) * sc.inv, y = (ty - sc.x0[1]) * sc.inv, z = (tz - sc.x0[2]) * sc.inv;
    const double m = fmax(fmax(fabs(x), fabs(y)), fabs(z));
    T.bad = !(m < 0x1p40) || isnan(x) || isnan(y) || isnan(z);
    T.fx = (float)x;
    T.fy = (float)y;
    T.fz = (float)z;
    int ex = 0;
    if (!T.bad) (void)frexp(m, &ex);
    T.st = ex > 0 ? ex : 0;
    const double s = __hiloint2double((1023 + fix64::kCoordBits - T.st) << 20, 0);
    T.x = T.bad ? 0 : __double2ll_rn(x * s);
    T.y = T.bad ? 0 : __double2ll_rn(y * s);
    T.z = T.bad ? 0 : __double2ll_rn(z * s);
    return T;
}

struct FxPairInfo {
    int c;               // rule: nearest physics node
    int e;               // pair exponent
    bool deferred;       // FP64
    float r0, rho;       // |D|, largest offset in the element
};

// Set-up of one pair: nearest node in FP32 with near / near-tie detection (the
// criteria of the mixed assembly), the pair's exponent, and D.
template <int NP, bool CPLX_K>
__device__ __forceinline__ FxPairInfo fx_pair(const float *r, const FxTarget &T, const FxWave &w, i64 &Dx, i64 &Dy,
                                              i64 &Dz) {
    FxPairInfo I;
    const i64 *cen = reinterpret_cast<const i64 *>(r + kHdrCen);
    Dx = (cen[0] >> T.st) - T.x;
    Dy = (cen[1] >> T.st) - T.y;
    Dz = (cen[2] >> T.st) - T.z;
    // FP32 D from the bits above 2^(29 - 59): 22 significant bits at the smallest
    // regular distance
    const float u = __int_as_float((127 - fix64::kCoordBits + 29 + T.st) << 23);
    const float fx = (float)(int)(Dx >> 29) * u, fy = (float)(int)(Dy >> 29) * u, fz = (float)(int)(Dz >> 29) * u;
    float d2[NP];
#pragma unroll
    for (int a = 0; a < NP; ++a) {
        const float ax = fx + r[kHdrNodes + 3 * a], ay = fy + r[kHdrNodes + 3 * a + 1],
                    az = fz + r[kHdrNodes + 3 * a + 2];
        d2[a] = ax * ax + ay * ay + az * az;
    }
    int c = 0;
    float b = d2[0];
#pragma unroll
    for (int a = 1; a < NP; ++a)
        if (d2[a] < b) {
            b = d2[a];
            c = a;
        }
    const float lim = b * (1.0f + 1e-5f);
    bool tie = false;
#pragma unroll
    for (int a = 0; a < NP; ++a) tie |= (a != c) && (d2[a] <= lim);
    const float r0f2 = fx * fx + fy * fy + fz * fz;
    const float near2 = r[kHdrNear2], rho = r[kHdrRho];
    const float r0 = sqrtf(r0f2);
    const float rmin = r0 * (1.0f - 1e-6f) - rho;
    I.c = c;
    I.r0 = r0;
    I.rho = rho;
    I.e = fix64::float_exp(rmin);
    I.deferred = T.bad || tie || r0f2 < near2 || 4.0f * b < near2 || !(r0 >= fix64::kRhoFactor * rho) ||
                 I.e < T.st + fix64::kMinExp || w.kx + I.e > fix64::kMaxTurnExp;
    if (CPLX_K)
        I.deferred |= !(fabsf(w.kl) * rho <= fix64::kMaxDampSpread) || w.kdx + I.e > fix64::kMaxDampExp;
    return I;
}


// Basis tables: per rule, group of four points and node the four values' limbs
// (two int4), zero beyond the rule's points.
constexpr int kGroup = 4;
constexpr int kInterleave = 2;   // points evaluated side by side
inline int phi_groups(int qmax) { return (qmax + kGroup - 1) / kGroup; }

// GW: per-element complex factors on G (the adjoint's element admittances), each
// against its own exponent; the unit of an entry of G then follows from the
// largest weight exponent times factor exponent among the node's elements.
struct FxFactors {
    const int4 *limbs;   // E
    const int *exps;     // E
    const int *nodes;    // N
};
template <int NP, bool CPLX_K, bool GW>
__global__ void __launch_bounds__(kThreads, 4)
assemble_fix64_kernel(const float *__restrict__ rec, int stride, int64_t E, int S,
                      const int4 *__restrict__ phi, int nphi, int ngroups, const __grid_constant__ RuleInfo ri,
                      const int4 *__restrict__ trig, const int2 *__restrict__ damp, const double *__restrict__ tgt, int64_t M,
                      double kre, double kim, int flags, longlong2 *__restrict__ F, longlong2 *__restrict__ G,
                      const uint32_t *__restrict__ kflags, double *__restrict__ Cpart,
                      int2 *__restrict__ defer, u64 *__restrict__ defer_count, unsigned int defer_cap,
                      int *__restrict__ over, const __grid_constant__ FxFactors gw, const __grid_constant__ FxScale sc,
                      unsigned long long *__restrict__ qpe_count, const double *__restrict__ kdev) {
    if (kdev) {   // wavenumber read from device memory (recorded sweeps)
        kre = kdev[0];
        kim = kdev[1];
    }
    extern __shared__ __align__(16) float smemf[];
    int4 *s_trig = reinterpret_cast<int4 *>(smemf);                              // 1024 entries
    int4 *s_val = s_trig + fix64::kTrigEntries;                                  // 2 kGroup x kThreads
    int4 *s_phi = s_val + 2 * kGroup * kThreads;                                      // nphi entries
    int2 *s_damp = reinterpret_cast<int2 *>(s_phi + nphi);                       // 256 entries (complex k)
    __shared__ RuleInfo s_ri;
    __shared__ FxWave s_wave;

    const int s = blockIdx.y;
    const int64_t e0 = (int64_t)s * E / S;
    const int64_t e1 = (int64_t)(s + 1) * E / S;
    const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const bool active = i < M;
    const bool doF = flags & BIE_F, doG = flags & BIE_G, doC = flags & BIE_C;

    double tx = 0, ty = 0, tz = 0;
    if (active) {
        tx = tgt[3 * i + 0];
        ty = tgt[3 * i + 1];
        tz = tgt[3 * i + 2];
    }
    const FxTarget T = fx_target(tx, ty, tz, sc);
    for (int t = threadIdx.x; t < fix64::kTrigEntries; t += kThreads) s_trig[t] = trig[t];
    for (int t = threadIdx.x; t < nphi; t += kThreads) s_phi[t] = phi[t];
    if (threadIdx.x == 0) {
        s_ri = ri;
        s_wave = fx_wave<CPLX_K>(kre, kim, sc);
    }
    if (CPLX_K)
        for (int t = threadIdx.x; t < fix64::kDampEntries; t += kThreads) s_damp[t] = damp[t];
    auto table = [s_trig](int j, Limb &c, Limb &sn) {
        const int4 v = s_trig[j];
        c = Limb{v.x, v.y};
        sn = Limb{v.z, v.w};
    };
    auto damp_table = [s_damp](int j) {
        const int2 v = s_damp[j];
        return Limb{v.x, v.y};
    };

    double cacc = 0.0;
    int over_at = fix64::kNoOverflow;
    unsigned long long nqpe = 0;
    __syncthreads();
    const FxWave wv = s_wave;
    char *Fi = reinterpret_cast<char *>(F + i), *Gi = reinterpret_cast<char *>(G + i);
    if (active) {
        for (int64_t pe = e0; pe < e1; ++pe) {
            const float *r = rec + pe * stride;
            const int *ir = reinterpret_cast<const int *>(r);
            fix64::Pair P;
            const FxPairInfo I = fx_pair<NP, CPLX_K>(r, T, wv, P.Dx, P.Dy, P.Dz);
            // (no flags: every node shared)
            const uint32_t fw = kflags ? __ldg(kflags + pe) : 0x00ff0000u;
            const int ej = ir[kHdrEj];
            const float *abs_nodes = r + kHdrNodes + 3 * NP;
            const int *node_ej = ir + kHdrNodes + 6 * NP;
            const int *nid = node_ej + NP;
            const int e = I.e;
            const int ejw = GW ? ej + __ldg(gw.exps + pe) : ej;   // of G
            int Q = 0;
            if (I.deferred) {   // no points here, but the pair may open or close entries
                u64 slot;
                if (fix64::defer_slot([=] { return atomicAdd(defer_count, 1ull); }, defer_cap, (int)pe, over_at, slot))
                    defer[slot] = make_int2((int)i, (int)pe);   // (else rescanned by the correction kernel)
            } else {
                const int qs = T.st + 2 - e;   // 2^(59 - st) units -> Q61 of 2^e
                P.Dx = (i64)((u64)P.Dx << qs);
                P.Dy = (i64)((u64)P.Dy << qs);
                P.Dz = (i64)((u64)P.Dz << qs);
                P.osh = min(63, 1 + e - ir[kHdrEo]);
                Q = s_ri.Q[I.c];
                nqpe += Q;
            }
            fix64::pair_wavenumber(P, wv.km, wv.kx, wv.ka, wv.kb, e);
            if (CPLX_K)
                fix64::pair_damping(P, wv.kd, wv.kdx, wv.kai, wv.kb, e,
                                    fix64::pair_base(wv.kl, I.r0, I.rho));
            const int4 *g4 = reinterpret_cast<const int4 *>(r + s_ri.off[I.c]);
            const int4 *phc = s_phi + (size_t)I.c * ngroups * NP * 2;
            i64 ce = 0;
            int q0 = 0;
            do {
                // kernel values of up to four points, through shared memory so that
                // one copy of the point sequence serves all of them
                for (int q = 0; q < kGroup; q += kInterleave) {
                    int4 vf[kInterleave], vg[kInterleave];
#pragma unroll
                    for (int j = 0; j < kInterleave; ++j) vf[j] = vg[j] = make_int4(0, 0, 0, 0);
                    if (q0 + q < Q) {
#pragma unroll
                        for (int j = 0; j < kInterleave; ++j) {
                            const int qj = min(q0 + q + j, Q - 1);
                            const int4 *w = g4 + 4 * qj;
                            const int4 A = __ldg(w), B = __ldg(w + 1), C4 = __ldg(w + 2);
                            const int2 D2 = __ldg(reinterpret_cast<const int2 *>(w + 3));
                            const bool on = q0 + q + j < Q;   // beyond the rule: weight zero
                            fix64::PointData g;
                            g.ox = fix64::make64(A.y, (unsigned)A.x);
                            g.oy = fix64::make64(A.w, (unsigned)A.z);
                            g.oz = fix64::make64(B.y, (unsigned)B.x);
                            g.nx = Limb{B.z, B.w};
                            g.ny = Limb{C4.x, C4.y};
                            g.nz = Limb{C4.z, C4.w};
                            g.jw = Limb{on ? D2.x : 0, on ? D2.y : 0};
                            const fix64::Point v = fix64::point<CPLX_K>(g, P, table, damp_table);
                            ce += v.tq;
                            const Limb a0 = fix64::split(v.Fr), a1 = fix64::split(v.Fi);
                            Limb a2 = fix64::split(v.Gr), a3 = fix64::split(v.Gi);
                            if (GW) {
                                const int4 f = __ldg(gw.limbs + pe);
                                const fix64::Values2 u = fix64::complex_mul(a2, a3, Limb{f.x, f.y}, Limb{f.z, f.w});
                                a2 = fix64::split(u.re);
                                a3 = fix64::split(u.im);
                            }
                            vf[j] = make_int4(a0.h, a0.l, a1.h, a1.l);
                            vg[j] = make_int4(a2.h, a2.l, a3.h, a3.l);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < kInterleave; ++j) {
                        s_val[(2 * (q + j)) * kThreads + threadIdx.x] = vf[j];
                        s_val[(2 * (q + j) + 1) * kThreads + threadIdx.x] = vg[j];
                    }
                }
                if (doF || doG) {
                    int4 vf[kGroup], vg[kGroup];
#pragma unroll
                    for (int q = 0; q < kGroup; ++q) {
                        vf[q] = s_val[(2 * q) * kThreads + threadIdx.x];
                        vg[q] = s_val[(2 * q + 1) * kThreads + threadIdx.x];
                    }
                    const bool open = q0 == 0, close = q0 + kGroup >= Q;
#pragma unroll 1
                    for (int a = 0; a < NP; ++a) {
                        const u64 off = fix64::column_bytes(nid[a], M);
                        longlong2 *pF = reinterpret_cast<longlong2 *>(Fi + off);
                        longlong2 *pG = reinterpret_cast<longlong2 *>(Gi + off);
                        const bool shared = (fw >> (16 + a)) & 1u;
                        const bool first = open && ((fw >> a) & 1u), last = close && ((fw >> (8 + a)) & 1u);
                        // the entry's sums so far, read ahead of the products
                        longlong2 vF = make_longlong2(0, 0), vG = vF;
                        if (!shared && !first) {
                            if (doF) vF = __ldcg(pF);
                            if (doG) vG = __ldcg(pG);
                        }
                        int p[2 * kGroup];
                        *reinterpret_cast<int4 *>(p) = phc[2 * a];
                        *reinterpret_cast<int4 *>(p + 4) = phc[2 * a + 1];
                        i64 fr = 0, fi = 0, gr = 0, gi = 0;       // high sums, Q55
                        const i64 half = (i64)1 << 31;
                        i64 frl = half, fil = half, grl = half, gil = half;   // cross sums
#pragma unroll
                        for (int q = 0; q < kGroup; ++q) {
                            const Limb ph{p[2 * q], p[2 * q + 1]};
                            const Limb a0{vf[q].x, vf[q].y}, a1{vf[q].z, vf[q].w}, a2{vg[q].x, vg[q].y},
                                a3{vg[q].z, vg[q].w};
                            fr = fix64::high(fr, a0, ph);
                            fi = fix64::high(fi, a1, ph);
                            gr = fix64::high(gr, a2, ph);
                            gi = fix64::high(gi, a3, ph);
                            frl = fix64::cross(frl, a0, ph);
                            fil = fix64::cross(fil, a1, ph);
                            grl = fix64::cross(grl, a2, ph);
                            gil = fix64::cross(gil, a3, ph);
                        }
                        const FxEntry en = fx_entry<CPLX_K>(T.fx, T.fy, T.fz, abs_nodes[3 * a], abs_nodes[3 * a + 1],
                                                            abs_nodes[3 * a + 2], wv);
                        const int fl = en.fl, de = e - (fl - 1);
                        const int dj = node_ej[a] - ej + sc.extra + (CPLX_K ? P.base - en.base : 0);
                        const int nw = GW ? __ldg(gw.nodes + nid[a]) : 0;
                        const int sg = max(0, (GW ? nw - ejw + sc.extra_w : dj) + de);
                        const int sf = max(0, dj + 2 * de + fix64::amplitude_exp(wv.kb, fl - 1) - P.fe);
                        vF.x += fix64::shift_right(fix64::fold(fr, frl), sf);
                        vF.y += fix64::shift_right(fix64::fold(fi, fil), sf);
                        vG.x += fix64::shift_right(fix64::fold(gr, grl), sg);
                        vG.y += fix64::shift_right(fix64::fold(gi, gil), sg);
                        if (shared) {
                            unsigned long long *uF = reinterpret_cast<unsigned long long *>(pF);
                            unsigned long long *uG = reinterpret_cast<unsigned long long *>(pG);
                            if (doF) {
                                atomicAdd(uF, (unsigned long long)vF.x);
                                atomicAdd(uF + 1, (unsigned long long)vF.y);
                            }
                            if (doG) {
                                atomicAdd(uG, (unsigned long long)vG.x);
                                atomicAdd(uG + 1, (unsigned long long)vG.y);
                            }
                            continue;
                        }
                        if (last) {   // final complex128 entries
                            const int adj = sc.pe + sc.extra - en.base;
                            vF = fx_complex<CPLX_K>(vF, fix64::entry_exp_f(node_ej[a], fl, wv.kb) + adj);
                            if (GW) vG = fx_complex<true>(vG, fix64::entry_exp_g(nw, fl) + sc.pe + sc.extra_w + sc.S);
                            else vG = fx_complex<CPLX_K>(vG, fix64::entry_exp_g(node_ej[a], fl) + adj + sc.S);
                        }
                        if (doF) *pF = vF;
                        if (doG) *pG = vG;
                    }
                }
                q0 += kGroup;
                phc += NP * 2;
            } while (q0 < Q);
            if (doC && Q > 0) cacc -= fx_double<false>(ce, ej - 2 * e - 57);
        }
    }
    if (active) {
        if (doC) Cpart[(int64_t)s * M + i] = cacc;
        over[(int64_t)s * M + i] = over_at;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nqpe += __shfl_down_sync(0xffffffffu, nqpe, o);
    if ((threadIdx.x & 31) == 0 && nqpe) atomicAdd(qpe_count, nqpe);
}

// Columns of the nodes shared between slices (and of untouched nodes; without a
// list, of all nodes): zeroed before the assembly, converted after it.
__global__ void fx_zero_kernel(const int32_t *__restrict__ fnode, int64_t nfix, int64_t M, longlong2 *__restrict__ F,
                               longlong2 *__restrict__ G) {
    const int64_t total = nfix * M;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = t / M;
        const size_t off = (size_t)(fnode ? fnode[n] : n) * (size_t)M + (size_t)(t - n * M);
        if (F) F[off] = make_longlong2(0, 0);
        if (G) G[off] = make_longlong2(0, 0);
    }
}

template <bool CPLX_K>
__global__ void fx_widen_kernel(const int32_t *__restrict__ fnode, int64_t nfix, const float4 *__restrict__ nodes,
                                const double *__restrict__ tgt, int64_t M, double kre, double kim,
                                const __grid_constant__ FxScale sc, longlong2 *__restrict__ F,
                                longlong2 *__restrict__ G, const int *__restrict__ gnodes,
                                const double *__restrict__ kdev) {
    if (kdev) {
        kre = kdev[0];
        kim = kdev[1];
    }
    __shared__ FxWave s_wave;
    if (threadIdx.x == 0) s_wave = fx_wave<CPLX_K>(kre, kim, sc);
    __syncthreads();
    const FxWave wv = s_wave;
    const int64_t total = nfix * M;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = t / M, i = t - n * M;
        const int64_t nd = fnode ? fnode[n] : n;
        const size_t off = (size_t)nd * (size_t)M + (size_t)i;
        const float4 x = nodes[nd];
        const float fx = (float)((tgt[3 * i] - sc.x0[0]) * sc.inv), fy = (float)((tgt[3 * i + 1] - sc.x0[1]) * sc.inv),
                    fz = (float)((tgt[3 * i + 2] - sc.x0[2]) * sc.inv);
        const FxEntry en = fx_entry<CPLX_K>(fx, fy, fz, x.x, x.y, x.z, wv);
        const int ej = __float_as_int(x.w), adj = sc.pe + sc.extra - en.base;
        if (F) F[off] = fx_complex<CPLX_K>(F[off], fix64::entry_exp_f(ej, en.fl, wv.kb) + adj);
        if (G && gnodes)
            G[off] = fx_complex<true>(G[off], fix64::entry_exp_g(gnodes[nd], en.fl) + sc.pe + sc.extra_w + sc.S);
        else if (G)
            G[off] = fx_complex<CPLX_K>(G[off], fix64::entry_exp_g(ej, en.fl) + adj + sc.S);
    }
}

// limbs and exponents of the element factors; nodes[j]: the largest exponent of
// weight times factor among node j's elements (3-node physics)
__global__ void fx_factor_kernel(const double2 *__restrict__ w, int64_t E, const float *__restrict__ rec, int stride,
                                 int4 *__restrict__ limbs, int *__restrict__ exps, int *__restrict__ nodes) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= E) return;
    const fix64::Factor f = fix64::element_factor(w[p].x, w[p].y);
    limbs[p] = make_int4(f.re.h, f.re.l, f.im.h, f.im.l);
    exps[p] = f.e;
    const int *r = reinterpret_cast<const int *>(rec + p * stride);
#pragma unroll
    for (int a = 0; a < 3; ++a) atomicMax(nodes + r[kHdrNodes + 7 * 3 + a], r[kHdrEj] + f.e);
}

template <int NP, bool CPLX_K>
__device__ __forceinline__ int fx_correct_pair(const Fp64View &v, int64_t i, int64_t p, const double *tgt, int64_t M,
                                               double kre, double kim, bool doF, bool doG, bool doC, double2 *F,
                                               double2 *G, double *Cnear, const double2 *gweight) {
    const double *r = v.rec + (size_t)p * v.stride;
    const double tx = tgt[3 * i], ty = tgt[3 * i + 1], tz = tgt[3 * i + 2];
    const int c = dev::nearest_node<NP>(r, tx, ty, tz);
    double fr[NP], fi[NP], gr[NP], gi[NP];
    const double ce = dev::element_fp64<NP, CPLX_K, dev::TrigFix>(r + v.ri.off[c], v.ri.Q[c],
                                                                  v.phi + (size_t)c * v.qmax * NP, tx, ty, tz, kre,
                                                                  kim, fr, fi, gr, gi, -1, dev::TrigFix{v.tab});
    if (gweight && doG) {
        const double2 w = gweight[p];
#pragma unroll
        for (int a = 0; a < NP; ++a) {
            const double t = gr[a] * w.x - gi[a] * w.y;
            gi[a] = gr[a] * w.y + gi[a] * w.x;
            gr[a] = t;
        }
    }
    const int32_t *nid = reinterpret_cast<const int32_t *>(r + v.nidx_off);
#pragma unroll
    for (int a = 0; a < NP; ++a) {
        const size_t off = (size_t)nid[a] * (size_t)M + (size_t)i;
        if (doF) {
            atomicAdd(&F[off].x, fr[a]);
            atomicAdd(&F[off].y, fi[a]);
        }
        if (doG) {
            atomicAdd(&G[off].x, gr[a]);
            atomicAdd(&G[off].y, gi[a]);
        }
    }
    if (doC) atomicAdd(&Cnear[i], ce);
    return v.ri.Q[c];
}

// FP64 integration of the deferred pairs, added to the finished entries.  Where
// the list was too short, every (row, slice) whose pairs did not all fit is
// gone through again from its first pair that found no place.
template <int NP, bool CPLX_K>
__global__ void __launch_bounds__(128)
fx_correct_kernel(const int2 *__restrict__ defer, const u64 *__restrict__ defer_count,
                  unsigned int defer_cap, const __grid_constant__ Fp64View v, const double *__restrict__ tgt,
                  int64_t M, double kre, double kim, int flags, double2 *__restrict__ F, double2 *__restrict__ G,
                  double *__restrict__ Cnear, const int *__restrict__ over, const float *__restrict__ rec, int stride,
                  int64_t E, int S, const __grid_constant__ FxScale sc, unsigned long long *__restrict__ qpe_count,
                  const double *__restrict__ kdev, const double2 *__restrict__ gweight) {
    if (kdev) {
        kre = kdev[0];
        kim = kdev[1];
    }
    const u64 total = *defer_count;
    const unsigned int n = (unsigned int)min(total, (u64)defer_cap);
    const bool doF = flags & BIE_F, doG = flags & BIE_G, doC = flags & BIE_C;
    unsigned long long nqpe = 0;
    for (unsigned int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        nqpe += fx_correct_pair<NP, CPLX_K>(v, defer[j].x, defer[j].y, tgt, M, kre, kim, doF, doG, doC, F, G,
                                                  Cnear, gweight);
    if (total > defer_cap) {
        const FxWave wv = fx_wave<CPLX_K>(kre, kim, sc);
        for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < M * S;
             j += (int64_t)gridDim.x * blockDim.x) {
            if (over[j] == fix64::kNoOverflow) continue;
            const int64_t s = j / M, i = j - s * M;
            const FxTarget T = fx_target(tgt[3 * i], tgt[3 * i + 1], tgt[3 * i + 2], sc);
            for (int64_t p = over[j]; p < (s + 1) * E / S; ++p) {
                i64 dx, dy, dz;
                if (!fx_pair<NP, CPLX_K>(rec + p * stride, T, wv, dx, dy, dz).deferred) continue;
                nqpe += fx_correct_pair<NP, CPLX_K>(v, i, p, tgt, M, kre, kim, doF, doG, doC, F, G, Cnear, gweight);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nqpe += __shfl_down_sync(0xffffffffu, nqpe, o);
    if ((threadIdx.x & 31) == 0 && nqpe) atomicAdd(qpe_count, nqpe);
}

inline unsigned stream_grid(const Ctx &c, int64_t total) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 16LL * c.num_sms));
}

bool on_nodes(const Ctx &c, const AssembleArgs &a) {
    return a.targets >= c.d_sources && a.targets + 3 * a.M <= c.d_sources + 3 * c.n_sources;
}

struct FxBuffers {
    double *Cpart, *Cnear;
    int2 *defer;
    u64 *dcount;
    unsigned int dcap;
    int *over;
};

template <int NP, bool CPLX>
void launch_np(Ctx &c, const AssembleArgs &a, const LaunchShape &sh, int spread, size_t smem, const FxBuffers &b) {
    const RecordLayout &L = c.lay;
    const Fix64Layout &X = c.xlay;
    RuleInfo ri{}, ri64{};
    for (int r = 0; r < L.R; ++r) {
        ri.Q[r] = ri64.Q[r] = L.Q[r];
        ri.off[r] = X.rule_off[r];
        ri64.off[r] = L.rule_off[r];
    }
    FxScale sc{};
    for (int k = 0; k < 3; ++k) sc.x0[k] = c.fx_origin[k];
    sc.S = c.fx_exp;
    sc.inv = std::ldexp(1.0, -c.fx_exp);
    sc.len = std::ldexp(1.0, c.fx_exp);
    sc.pe = c.fx_phi_exp;
    sc.extra = c.fx_extra;
    sc.rho_max = c.fx_rho_max;
    FxFactors gw{};
    if (a.g_weight && (a.flags & BIE_G)) {
        const size_t E = (size_t)c.n_elements, N = (size_t)c.n_sources;
        int4 *limbs = static_cast<int4 *>(c.scratch(kScratchFxWeight, E * 20 + N * 4));
        int *exps = reinterpret_cast<int *>(limbs + E), *nodes = exps + E;
        BIE_CUDA(cudaMemsetAsync(nodes, 0xc0, N * 4, c.stream));   // far below every exponent
        fx_factor_kernel<<<(unsigned)((E + 255) / 256), 256, 0, c.stream>>>(
            reinterpret_cast<const double2 *>(a.g_weight), c.n_elements, c.d_xrecords, X.stride, limbs, exps, nodes);
        BIE_CUDA(cudaGetLastError());
        ++c.kernel_launches;
        gw = FxFactors{limbs, exps, nodes};
        sc.extra_w = c.fx_extra_w;
    }
    const Fp64View v{c.d_records, L.stride, L.nidx_off, c.d_phi, L.qmax, ri64, c.d_xtrig};
    const int level = sh.level, S = spread ? spread : 1 << level;
    const int64_t E = c.n_elements, nfix = spread ? c.n_sources : c.k2_nfix[level];
    longlong2 *F = (a.flags & BIE_F) ? reinterpret_cast<longlong2 *>(a.F) : nullptr;
    longlong2 *G = (a.flags & BIE_G) ? reinterpret_cast<longlong2 *>(a.G) : nullptr;
    const int32_t *fnode = spread ? nullptr : c.d_k2_fix + c.k2_fix_off[level];
    if (nfix > 0 && (F || G)) {
        fx_zero_kernel<<<stream_grid(c, nfix * a.M), 256, 0, c.stream>>>(fnode, nfix, a.M, F, G);
        BIE_CUDA(cudaGetLastError());
        ++c.kernel_launches;
    }
    auto kern = assemble_fix64_kernel<NP, CPLX, false>;
    if constexpr (NP == 3 && !CPLX)
        if (gw.limbs) kern = assemble_fix64_kernel<NP, CPLX, true>;
    BIE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((unsigned)((a.M + kThreads - 1) / kThreads), (unsigned)S);
    cudaEvent_t t0 = c.timer_begin();
    kern<<<grid, kThreads, smem, c.stream>>>(
        c.d_xrecords, X.stride, E, S, reinterpret_cast<const int4 *>(c.d_xphi), L.R * phi_groups(L.qmax) * NP * 2,
        phi_groups(L.qmax), ri,
        reinterpret_cast<const int4 *>(c.d_xtrig),
        reinterpret_cast<const int2 *>(c.d_xtrig + 4 * fix64::kTrigEntries), a.targets, a.M, a.k_re, a.k_im, a.flags, F, G,
        spread ? nullptr : c.d_k2_flags + (size_t)level * E, b.Cpart, b.defer, b.dcount, b.dcap, b.over, gw, sc, c.d_qpe, a.k_dev);
    BIE_CUDA(cudaGetLastError());
    c.timer_end(t0);
    ++c.kernel_launches;
    if (nfix > 0 && (F || G)) {
        fx_widen_kernel<CPLX><<<stream_grid(c, nfix * a.M), 256, 0, c.stream>>>(
            fnode, nfix, reinterpret_cast<const float4 *>(c.d_xnodes), a.targets, a.M, a.k_re, a.k_im, sc, F, G,
            gw.nodes, a.k_dev);
        BIE_CUDA(cudaGetLastError());
        ++c.kernel_launches;
    }
    auto corr = fx_correct_kernel<NP, CPLX>;
    // (far from the surface every pair can be here: 30000 points at 10^5 sizes 96 ms
    // with 4 blocks per SM, 84 with 16, the FP64 kernel alone 95; on the surface a few
    // per cent of the pairs)
    const int64_t most = (a.M * E + 127) / 128;
    corr<<<(unsigned)std::min<int64_t>(most, (on_nodes(c, a) ? 4LL : 16LL) * c.num_sms), 128, 0, c.stream>>>(
        b.defer, b.dcount, b.dcap, v, a.targets, a.M, a.k_re, a.k_im, a.flags, reinterpret_cast<double2 *>(F),
        reinterpret_cast<double2 *>(G), b.Cnear, b.over, c.d_xrecords, X.stride, E, S, sc, c.d_qpe, a.k_dev,
        reinterpret_cast<const double2 *>(a.g_weight));
    BIE_CUDA(cudaGetLastError());
    ++c.kernel_launches;
}

// ---- records ------------------------------------------------------------------
// Built on the device from the FP64 records: one thread per element (thousands of
// elements, a few hundred FP64 operations each).  On the host, one thread, this
// made a context 18 to 44 % more expensive (rigid sphere P2, 5780 elements: 5.9 ms).
struct FxBuild {
    double x0[3], inv, area;      // origin, 2^-S, 2^-2S / 4 pi
    int NP, R, qmax, pe;          // pe: basis values are stored times 2^-pe
    int stride64, stride;
    int Q[kMaxRules], off64[kMaxRules], off[kMaxRules];
};
struct FxSummary {                // (non-negative doubles and floats compare as integers)
    unsigned long long reach, reach_all;
    unsigned int rho, bad, small, unused;
};

__device__ __forceinline__ i64 fx_fixed(double h, double l, double scale) {
    return __double2ll_rn(h * scale) + __double2ll_rn(l * scale);
}
__device__ __forceinline__ void fx_put64(int *w, i64 v) {
    w[0] = fix64::lo32(v);
    w[1] = fix64::hi32(v);
}
__device__ __forceinline__ void fx_put_limbs(int *w, i64 v) {
    const Limb l = fix64::split(v);
    w[0] = l.h;
    w[1] = l.l;
}
// a - b = s + err exactly
__device__ __forceinline__ double fx_diff(double a, double b, double &err) {
    const double s = __dsub_rn(a, b), bb = __dsub_rn(s, a);
    err = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(-b, bb));
    return s;
}

// corners: the three corner vertices of every element.  nodes: largest weight
// exponent per node; reach: max over rules of sum |jw| |phi| in 2^(ej + pe).
__global__ void __launch_bounds__(64)
fx_build_kernel(const double *__restrict__ rec64, const double *__restrict__ corners, const double *__restrict__ phi,
                int64_t E, const __grid_constant__ FxBuild b, int *__restrict__ rec, int *__restrict__ nodes,
                double *__restrict__ reach, FxSummary *__restrict__ sum, const int32_t *__restrict__ nidx, int nidx_off) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= E) return;
    const int NP = b.NP;
    const double *R0 = rec64 + p * b.stride64, *V = corners + 9 * p;
    int *w = rec + p * b.stride;
    float *wf = reinterpret_cast<float *>(w);
    double cen[3], hmax = 0.0;
    for (int k = 0; k < 3; ++k) {
        cen[k] = __dadd_rn(__dadd_rn(__ddiv_rn(V[k], 3.0), __ddiv_rn(V[3 + k], 3.0)), __ddiv_rn(V[6 + k], 3.0));
        double err;
        const double s = fx_diff(cen[k], b.x0[k], err);
        fx_put64(w + kHdrCen + 2 * k, fx_fixed(s * b.inv, err * b.inv, 0x1p59));
    }
    for (int a = 0; a < 3; ++a) {
        const double *A = V + 3 * a, *B = V + 3 * ((a + 1) % 3);
        double d2 = 0.0;
        for (int k = 0; k < 3; ++k) {
            const double d = (A[k] - B[k]) * b.inv;
            d2 += d * d;
        }
        hmax = fmax(hmax, d2);
    }
    wf[kHdrNear2] = (float)hmax;
    double rho2 = 0.0, omax = 0.0, jmax = 0.0, jsum = 0.0;
    for (int a = 0; a < NP; ++a) {
        double d2 = 0.0;
        for (int k = 0; k < 3; ++k) {
            const double x = R0[3 * a + k], d = (x - cen[k]) * b.inv;
            d2 += d * d;
            wf[kHdrNodes + 3 * a + k] = (float)d;
            wf[kHdrNodes + 3 * NP + 3 * a + k] = (float)((x - b.x0[k]) * b.inv);
        }
        rho2 = fmax(rho2, d2);
    }
    for (int r = 0; r < b.R; ++r) {
        const int Q = b.Q[r];
        const double *g = R0 + b.off64[r];
        double js = 0.0;
        for (int q = 0; q < Q; ++q) {
            double d2 = 0.0;
            for (int k = 0; k < 3; ++k) {
                const double d = (g[k * Q + q] - cen[k]) * b.inv;
                d2 += d * d;
                omax = fmax(omax, fabs(d));
            }
            rho2 = fmax(rho2, d2);
            const double j = fabs(g[6 * Q + q]) * b.area;
            jmax = fmax(jmax, j);
            js += j;
        }
        jsum = fmax(jsum, js);
    }
    const float rho = (float)(sqrt(rho2) * (1.0 + 1e-6));
    wf[kHdrRho] = rho;
    atomicMax(&sum->rho, __float_as_uint(rho));
    // (regular pairs of such elements lie closer than the fixed range: FP64)
    if (ldexpf(fix64::kRhoFactor * rho, 1 - fix64::kMinExp) < 1.0f) atomicAdd(&sum->small, 1u);
    int eo = 0, je = 0;
    (void)frexp(omax > 0 ? omax * (1.0 + 1e-9) : 0x1p-60, &eo);
    (void)frexp(jmax > 0 ? jmax * 1.01 : 0x1p-200, &je);
    while (ldexp(jsum, -je) > 8.0) ++je;   // sums over a rule: |sum t| < 8 * 4 2^57
    if (je < -900) {
        sum->bad = 1;
        return;
    }
    w[kHdrEj] = je;
    w[kHdrEo] = eo;
    const double so = ldexp(1.0, 62 - eo), sj = ldexp(b.area, 63 - je);
    for (int r = 0; r < b.R; ++r) {
        const int Q = b.Q[r];
        const double *g = R0 + b.off64[r];
        for (int q = 0; q < Q; ++q) {
            int *P = w + b.off[r] + kPointWords * q;
            for (int k = 0; k < 3; ++k) {
                double err;
                const double s = fx_diff(g[k * Q + q], cen[k], err);
                fx_put64(P + 2 * k, fx_fixed(s * b.inv, err * b.inv, so));
                fx_put_limbs(P + 6 + 2 * k, __double2ll_rn(g[(3 + k) * Q + q] * 0x1p61));
            }
            fx_put_limbs(P + 12, __double2ll_rn(g[6 * Q + q] * sj));
        }
    }
    const int32_t *nid = nidx + 2 * (p * b.stride64 + nidx_off);
    for (int a = 0; a < NP; ++a) {
        double best = 0.0;
        for (int r = 0; r < b.R; ++r) {
            double s = 0.0;
            for (int q = 0; q < b.Q[r]; ++q)
                s += fabs(R0[b.off64[r] + 6 * b.Q[r] + q] * phi[((int64_t)r * b.qmax + q) * NP + a]);
            best = fmax(best, s);
        }
        reach[p * NP + a] = ldexp(best * b.area, -je - b.pe);
        w[kHdrNodes + 7 * NP + a] = nid[a];
        atomicMax(nodes + nid[a], je);
    }
}

// The node's weight exponent into every record, and the sums of the reaches per
// node: in units of that exponent, and each in its own (element factors may make
// any contribution the node's largest).
__global__ void fx_build_nodes_kernel(int64_t E, const __grid_constant__ FxBuild b, int *__restrict__ rec,
                                      const int *__restrict__ nodes, const double *__restrict__ reach,
                                      double *__restrict__ sums, int64_t N) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= E * b.NP) return;
    const int64_t p = t / b.NP;
    const int a = (int)(t - p * b.NP);
    int *w = rec + p * b.stride;
    const int nd = w[kHdrNodes + 7 * b.NP + a], je = nodes[nd];
    w[kHdrNodes + 6 * b.NP + a] = je;
    atomicAdd(sums + nd, ldexp(reach[t], w[kHdrEj] - je));
    atomicAdd(sums + N + nd, reach[t]);
}

__global__ void fx_build_finish_kernel(int64_t N, const __grid_constant__ FxBuild b, const double *__restrict__ src,
                                       const int *__restrict__ nodes, const double *__restrict__ sums,
                                       float4 *__restrict__ xnodes, FxSummary *__restrict__ sum) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N) return;
    const int je = nodes[j];
    xnodes[j] = make_float4((float)((src[3 * j] - b.x0[0]) * b.inv), (float)((src[3 * j + 1] - b.x0[1]) * b.inv),
                            (float)((src[3 * j + 2] - b.x0[2]) * b.inv), __int_as_float(je == INT_MIN ? 0 : je));
    atomicMax(&sum->reach, (unsigned long long)__double_as_longlong(sums[j]));
    atomicMax(&sum->reach_all, (unsigned long long)__double_as_longlong(sums[N + j]));
}

}  // namespace

// e^{2 pi i j / 1024} and 2^(-j / 256) as Q62 limbs (constants: built once; the
// extended arithmetic is software on some hosts)
static const std::vector<int32_t> &unit_tables() {
    static const std::vector<int32_t> table = [] {
        const int n = fix64::kTrigEntries;
        std::vector<int32_t> t((size_t)4 * n + 2 * fix64::kDampEntries);
        const long double pi = 3.141592653589793238462643383279502884L;
        auto put = [](int32_t *w, long double x) {
            const fix64::Limb s = fix64::split((long long)std::llrint(std::ldexp(x, 62)));
            w[0] = s.h;
            w[1] = s.l;
        };
        for (int j = 0; j < n; ++j) {
            put(&t[4 * j], std::cos(2.0L * pi * j / n));
            put(&t[4 * j + 2], std::sin(2.0L * pi * j / n));
        }
        for (int j = 0; j < fix64::kDampEntries; ++j)
            put(&t[4 * n + 2 * j], std::exp2(-(long double)j / fix64::kDampEntries));
        return t;
    }();
    return table;
}

// Records of the fixed-point kernels from the FP64 ones (c.d_records).
void build_fix64_records(Ctx &c) {
    const RecordLayout &L = c.lay;
    Fix64Layout &X = c.xlay;
    X = Fix64Layout{};
    const int NP = L.NP;
    const int64_t E = c.n_elements, N = c.n_sources;
    c.fx_ok = false;
    const std::vector<int32_t> &trig = unit_tables();   // (the near pairs of every precision use them)
    BIE_CUDA(cudaMalloc(&c.d_xtrig, trig.size() * 4));
    BIE_CUDA(cudaMemcpy(c.d_xtrig, trig.data(), trig.size() * 4, cudaMemcpyHostToDevice));
    // scaled coordinates (x - x0) 2^-S with the largest in [1/2, 1).  x0 is zero
    // unless the mesh lies far from the origin for its size, where the
    // subtraction is exact for targets near the mesh.
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    auto span = [&](const std::vector<double> &v) {
        for (size_t j = 0; j < v.size(); j += 3)
            for (int k = 0; k < 3; ++k) {
                lo[k] = std::min(lo[k], v[j + k]);
                hi[k] = std::max(hi[k], v[j + k]);
            }
    };
    span(c.coords);
    span(c.sources);
    double ext = 0.0, top = 0.0;
    for (int k = 0; k < 3; ++k) ext = std::max(ext, hi[k] - lo[k]);
    for (int k = 0; k < 3; ++k) {
        const double mid = 0.5 * (lo[k] + hi[k]);
        c.fx_origin[k] = std::fabs(mid) > 4.0 * ext ? mid : 0.0;
        top = std::max(top, std::max(std::fabs(lo[k] - c.fx_origin[k]), std::fabs(hi[k] - c.fx_origin[k])));
    }
    if (!(top > 0x1p-300 && top < 0x1p300)) return;   // such meshes stay with the FP64 kernel
    (void)std::frexp(top, &c.fx_exp);
    const double inv = std::ldexp(1.0, -c.fx_exp);
    auto put_limbs = [](int32_t *w, long long v) {
        const fix64::Limb s = fix64::split(v);
        w[0] = s.h;
        w[1] = s.l;
    };

    int off = kHdrNodes + 6 * NP + 2 * NP;
    off = (off + 3) & ~3;
    for (int r = 0; r < L.R; ++r) {
        X.rule_off[r] = off;
        off += kPointWords * L.Q[r];
    }
    X.stride = off;

    // basis scale: |phi| 2^-pe <= 1
    double pmax = 0.0;
    for (double p : c.phi) pmax = std::max(pmax, std::fabs(p));
    c.fx_phi_exp = 0;
    while (std::ldexp(pmax, -c.fx_phi_exp) > 1.0) ++c.fx_phi_exp;
    const int ng = phi_groups(L.qmax);
    std::vector<int32_t> phi((size_t)L.R * ng * NP * 2 * kGroup, 0);
    for (int r = 0; r < L.R; ++r)
        for (int q = 0; q < L.Q[r]; ++q)
            for (int a = 0; a < NP; ++a)
                put_limbs(&phi[((((size_t)r * ng + q / kGroup) * NP + a) * kGroup + q % kGroup) * 2],
                          (long long)std::llrint(std::ldexp(c.phi[((size_t)r * L.qmax + q) * NP + a], 61 - c.fx_phi_exp)));

    FxBuild b{};
    for (int k = 0; k < 3; ++k) b.x0[k] = c.fx_origin[k];
    b.inv = inv;
    b.area = inv * inv * dev::kInv4Pi;
    b.NP = NP;
    b.R = L.R;
    b.qmax = L.qmax;
    b.pe = c.fx_phi_exp;
    b.stride64 = L.stride;
    b.stride = X.stride;
    for (int r = 0; r < L.R; ++r) {
        b.Q[r] = L.Q[r];
        b.off64[r] = L.rule_off[r];
        b.off[r] = X.rule_off[r];
    }
    std::vector<double> corners((size_t)9 * E);
    for (int64_t p = 0; p < E; ++p)
        for (int a = 0; a < 3; ++a)
            for (int k = 0; k < 3; ++k)
                corners[9 * p + 3 * a + k] = c.coords[3 * (int64_t)c.topo[c.NS * c.order[p] + a] + k];
    // temporary: corners, reaches, sums per node, summary, exponents per node
    struct Temp {
        char *p = nullptr;
        ~Temp() { cudaFree(p); }
    } tmp;
    const size_t nc = corners.size() * 8, nr = (size_t)E * NP * 8, ns = (size_t)2 * N * 8;
    FxSummary sum{};
    try {
        BIE_CUDA(cudaMalloc(&tmp.p, nc + nr + ns + sizeof(FxSummary) + (size_t)N * 4));
        BIE_CUDA(cudaMalloc(&c.d_xrecords, (size_t)E * X.stride * 4));
        BIE_CUDA(cudaMalloc(&c.d_xphi, phi.size() * 4));
        BIE_CUDA(cudaMalloc(&c.d_xnodes, (size_t)N * 16));
    } catch (const Error &e) {   // no room: the other kernels do without
        if (e.code != BIE_ERR_NOMEM) throw;
        cudaGetLastError();
        cudaFree(c.d_xrecords);
        cudaFree(c.d_xphi);
        c.d_xrecords = nullptr;
        c.d_xphi = nullptr;
        return;
    }
    double *d_corners = reinterpret_cast<double *>(tmp.p), *d_reach = d_corners + 9 * E, *d_sums = d_reach + E * NP;
    FxSummary *d_sum = reinterpret_cast<FxSummary *>(d_sums + 2 * N);
    int *d_nodes = reinterpret_cast<int *>(d_sum + 1);
    // (all on the default stream: in order with the uploads of the FP64 records)
    BIE_CUDA(cudaMemcpy(d_corners, corners.data(), nc, cudaMemcpyHostToDevice));
    BIE_CUDA(cudaMemcpy(c.d_xphi, phi.data(), phi.size() * 4, cudaMemcpyHostToDevice));
    BIE_CUDA(cudaMemsetAsync(d_sums, 0, ns + sizeof(FxSummary), 0));
    BIE_CUDA(cudaMemsetAsync(c.d_xrecords, 0, (size_t)E * X.stride * 4, 0));
    const std::vector<int> none((size_t)N, INT_MIN);
    BIE_CUDA(cudaMemcpy(d_nodes, none.data(), (size_t)N * 4, cudaMemcpyHostToDevice));
    int *rec = reinterpret_cast<int *>(c.d_xrecords);
    fx_build_kernel<<<(unsigned)((E + 63) / 64), 64>>>(c.d_records, d_corners, c.d_phi, E, b, rec, d_nodes, d_reach,
                                                       d_sum, reinterpret_cast<const int32_t *>(c.d_records),
                                                       L.nidx_off);
    BIE_CUDA(cudaGetLastError());
    fx_build_nodes_kernel<<<(unsigned)((E * NP + 255) / 256), 256>>>(E, b, rec, d_nodes, d_reach, d_sums, N);
    BIE_CUDA(cudaGetLastError());
    fx_build_finish_kernel<<<(unsigned)((N + 255) / 256), 256>>>(N, b, c.d_sources, d_nodes, d_sums,
                                                                 reinterpret_cast<float4 *>(c.d_xnodes), d_sum);
    BIE_CUDA(cudaGetLastError());
    BIE_CUDA(cudaMemcpy(&sum, d_sum, sizeof(sum), cudaMemcpyDeviceToHost));
    if (sum.bad) return;
    std::memcpy(&c.fx_rho_max, &sum.rho, 4);
    c.fx_small = sum.small;
    // entries hold |sum| <= 4 sqrt(2) 2^55 sum of the reaches: below 2^62 (a factor's
    // modulus is up to sqrt(2) of its unit: G with factors is below half of F's bound)
    auto extra_of = [](unsigned long long bits) {
        double worst;
        std::memcpy(&worst, &bits, 8);
        int x = 0;
        while (std::ldexp(worst * 5.7, -x) > 127.0) ++x;
        return x;
    };
    c.fx_extra = extra_of(sum.reach);
    c.fx_extra_w = extra_of(sum.reach_all);
    c.fx_ok = true;
}

// Small phases stay in floating point: values here are good to 2^-55 of the modulus,
// but with k r small the imaginary parts, k and k^3 times the real ones, are
// results of their own.  FP64 rounds k r cos(k r) - sin(k r) to 2^-53 k r, so at
// k r = 1/4 both are alike; below that the fixed-point parts lose: on the unit
// sphere (2^S = 2) Im F and Im G differ from plain FP64 by 2e-14 and 2e-16 at k = 0.3,
// 6e-13 and 5e-16 at 0.1, 6e-10 and 5e-15 at 0.01.
bool fix64_small_phase(const Ctx &c, double k_re) {
    return k_re != 0.0 && std::fabs(k_re) * std::ldexp(1.0, c.fx_exp) < 0.25;
}

static bool fix64_covers(const Ctx &c, const AssembleArgs &a) {
    if (!c.fx_ok || a.taylor_m >= 0 || (a.g_weight && !a.g_weight_bounded)) return false;
    if (a.k_dev && !(a.k_abs_max > 0)) return false;   // no bound on |k|
    if (a.M > INT32_MAX) return false;   // rows are 32-bit in the list of deferred pairs
    const bool cplx = a.k_im != 0.0;
    if (a.g_weight && (c.lay.NP != 3 || cplx)) return false;   // (the adjoint: 3-node physics, real k)
    // wavenumbers whose phase or damping over the mesh or an element leaves the
    // fixed-point ranges for many pairs stay with the FP64 kernel
    const double bound = a.k_dev ? a.k_abs_max : 0.0, len = std::ldexp(1.0, c.fx_exp);
    const double kr = std::max(std::fabs(a.k_re), bound) * len, ki = cplx ? std::max(std::fabs(a.k_im), bound) * len : 0.0;
    if (!(kr < 500.0 && ki < 100.0 && ki * c.fx_rho_max * 1.45 < fix64::kMaxDampSpread)) return false;
    // (C does not depend on k)
    return !(a.flags & (BIE_F | BIE_G)) || !fix64_small_phase(c, a.k_dev ? a.k_re_min : a.k_re);
}

// Where the double-float kernel is available (BIE_PREC_DF64), the fixed-point one
// takes the node rows of 4-point rules: its entries cost less, its points more.
// Against the double-float kernel, 320 to 8000 elements: 4-point rules 1.09 to
// 1.65 times as fast (complex k 1.03 to 1.5, 0.92 to 1.3 on 320 elements); 9- and
// 16-point rules 0.85 to 1.15 (complex k 0.57 to 1.14); targets off the surface,
// where C takes a pass of its own, 0.6 to 1.2 (complex k 0.35 to 1.2).  On graded
// meshes the pairs among elements below 2^-9 of the mesh go to FP64: 2562 nodes with
// element sizes over a factor of 1000 3.2 and 4.8 ms (36 and 69 % of the elements
// small), the double-float kernel 1.9.
bool fix64_takes(const Ctx &c, const AssembleArgs &a, bool df64) {
    if (df64 && 8 * (int64_t)c.fx_small > c.n_elements) return false;
    if (df64 && !(on_nodes(c, a) && c.lay.Q[0] <= 4 && (a.k_im == 0.0 || c.n_elements >= 512))) return false;
    return fix64_covers(c, a);
}

bool launch_assemble_fix64(Ctx &c, const AssembleArgs &args, bool df64) {
    if (!fix64_takes(c, args, df64)) return false;
    AssembleArgs a = args;
    const bool cplx = a.k_im != 0.0;
    // The finest slicing with at least four elements per slice: blocks differ in
    // cost (near pairs leave points out, midpoint rules add some), so many small
    // ones even out.  Step at 128 / 64 / 32 slices: pulsating sphere 20.8 / 21.2 /
    // 22.0 ms, rigid sphere P2 11.3 / 11.4 / 12.0, 5762 nodes P2 3.20 / 3.30 / 3.55,
    // 362 nodes with 16-point rules 0.22 / 0.29 / 0.40.
    int level = 0;
    while (level + 1 < kMaxLevels && (c.n_elements >> (level + 1)) >= 4) ++level;
    // Few rows do not fill the SMs with that (a pair takes microseconds, one after
    // the other on its thread): four waves of blocks, on slices down to single
    // elements, with every node shared (integer atomics).  8000 elements, 40 / 700 /
    // 1333 / 2600 rows against the slices above: P2 with 16-point rules 2.00 -> 0.56,
    // 6.0 -> 4.1, 8.4 -> 7.3, 14.4 -> 13.9 ms, P1 with 4-point rules 0.29 -> 0.13, 0.84
    // -> 0.71, 1.33 -> 1.26, 2.29 -> 2.36; without shared nodes, whose entries need no
    // atomics otherwise, 0.29 -> 0.15, 130 rows 0.37 -> 0.32, but 300 rows 0.45 -> 0.54.
    const int64_t tiles = (a.M + kThreads - 1) / kThreads, resident = 4LL * c.num_sms;
    // (BIE_PREC_DF64 keeps its tunable slices)
    const bool few = !df64 && tiles << level <= (c.k2_nfix[level] > 0 ? 3 * resident : resident / 2);
    const int spread = few ? (int)std::min<int64_t>(c.n_elements, 4 * resident / tiles) : 0;
    // list of deferred pairs, counter, C of these; and per (slice, row) the C partial
    // sums and the overflow marks: up to 2 KB a row, where the FP64 kernel needs 8 bytes
    // a slice.  It takes over where the device has no room for that beside the outputs.
    const unsigned int dcap = (unsigned int)std::min<int64_t>(a.M * 64 + 4096, (int64_t)1 << 30);
    const size_t dbytes = (size_t)dcap * sizeof(int2);
    const size_t part_row = (size_t)(spread ? spread : 1 << level) * (sizeof(double) + sizeof(int));
    if ((a.flags & (BIE_F | BIE_G)) || on_nodes(c, a)) {
        if (!c.scratch_fits(kScratchDefer, dbytes + 256 + (size_t)a.M * 8)) return false;
        if (!c.scratch_fits(kScratchCpart, part_row * a.M)) {
            c.drop_scratch(kScratchDefer);
            return false;
        }
    }
    // C at points off the surface cancels to the quadrature error, where any other
    // rounding would show: it keeps the FP64 operations
    struct Join {   // the call's stream waits for the side stream, whatever happens in between
        Ctx &c;
        bool on = false;
        ~Join() {
            if (on) cudaStreamWaitEvent(c.stream, c.side_ev[1], 0);
        }
    } join{c};
    if ((a.flags & BIE_C) && !on_nodes(c, a)) {
        // beside the fixed-point kernel (side streams are made outside captures)
        const bool beside = (a.flags & (BIE_F | BIE_G)) && (c.side_stream || !c.capturing);
        launch_field_c_fp64(c, a.targets, a.M, a.C, beside);
        join.on = beside;
        a.flags &= ~BIE_C;
    }
    if (!(a.flags & (BIE_F | BIE_G | BIE_C))) return true;
    const RecordLayout &L = c.lay;
    FxBuffers b{};
    b.dcap = dcap;
    char *dbuf = static_cast<char *>(c.scratch(kScratchDefer, dbytes + 256 + (size_t)a.M * 8));
    b.defer = reinterpret_cast<int2 *>(dbuf);
    b.dcount = reinterpret_cast<u64 *>(dbuf + dbytes);
    b.Cnear = reinterpret_cast<double *>(dbuf + dbytes + 256);
    auto reset = [&] { BIE_CUDA(cudaMemsetAsync(dbuf + dbytes, 0, 256 + (size_t)a.M * 8, c.stream)); };
    reset();

    auto run = [&](const LaunchShape &sh) {
        const int S = spread ? spread : 1 << sh.level;
        // phase table, point values of the block's threads, basis tables
        const size_t smem = ((size_t)fix64::kTrigEntries + 2 * kGroup * kThreads +
                             (size_t)L.R * phi_groups(L.qmax) * L.NP * 2) * 16 +
                            (cplx ? fix64::kDampEntries * 8 : 0);
        // per (slice, row): the C partial sums, then the overflow marks
        const size_t cp = (size_t)S * a.M * sizeof(double);
        char *part = static_cast<char *>(c.scratch(kScratchCpart, cp + (size_t)S * a.M * sizeof(int)));
        b.Cpart = reinterpret_cast<double *>(part);
        b.over = reinterpret_cast<int *>(part + cp);
        if (L.NP == 1) {
            if (cplx) launch_np<1, true>(c, a, sh, spread, smem, b);
            else launch_np<1, false>(c, a, sh, spread, smem, b);
        } else if (L.NP == 3) {
            if (cplx) launch_np<3, true>(c, a, sh, spread, smem, b);
            else launch_np<3, false>(c, a, sh, spread, smem, b);
        } else {
            if (cplx) launch_np<6, true>(c, a, sh, spread, smem, b);
            else launch_np<6, false>(c, a, sh, spread, smem, b);
        }
        if (a.flags & BIE_C) launch_reduce_c(c, b.Cpart, S, b.Cnear, a.M, a.C, nullptr, true);
    };
    // (records are read through L1: the chunk is the double-float kernel's, which
    // shares the tuned shape)
    const int chunk0 = (int)std::max<size_t>(1, std::min<size_t>(32, (32u << 10) / ((size_t)c.dlay.stride * sizeof(float))));
    const LaunchShape base{level, chunk0, kThreads};
    ShapeAxes ax;
    for (int l = level - 1; l <= level + 1; ++l)
        if (l >= 0 && l < kMaxLevels && (int64_t(1) << l) <= c.n_elements) ax.levels.push_back(l);
    run(df64 ? resolve_shape(c, kShapeK9, a.M, base, ax, run, reset) : base);
    return true;
}

}  // namespace bie
