// Drives the quadrature points of bie_fix64.cuh with complex wavenumbers and with
// phases of many turns on the host against long double: prints whether every
// table index lay inside its table, and the largest error of F and G over random
// regular pairs as a multiple of its bound.  Arguments: seed, binary exponent of the
// largest phase in turns, 1 for complex k.
#include "bie_fix64.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace bie::fix64;
typedef long double Q;

static i64 fixed(Q x, int n) { return (i64)llrintl(ldexpl(x, n)); }

template <bool CPLX>
static double run(unsigned long long seed, int turns, bool &inside) {
    std::mt19937_64 gen(seed);
    auto U = [&] { return (double)(gen() >> 11) * 0x1p-53; };
    const Q pi = 3.141592653589793238462643383279502884L, log2e = 1.442695040888963407359924681001892137L;
    static Limb tc[kTrigEntries], ts[kTrigEntries], td[kDampEntries];
    for (int j = 0; j < kTrigEntries; ++j) {
        tc[j] = split(fixed(cosl(2 * pi * j / kTrigEntries), 62));
        ts[j] = split(fixed(sinl(2 * pi * j / kTrigEntries), 62));
    }
    for (int j = 0; j < kDampEntries; ++j) td[j] = split(fixed(exp2l(-(Q)j / kDampEntries), 62));
    auto trig = [&](int j, Limb &c, Limb &s) {
        inside = inside && j >= 0 && j < kTrigEntries;
        c = tc[j & (kTrigEntries - 1)];
        s = ts[j & (kTrigEntries - 1)];
    };
    auto damp = [&](int j) {
        inside = inside && j >= 0 && j < kDampEntries;
        return td[j & (kDampEntries - 1)];
    };
    double worst = 0.0;
    int done = 0;
    while (done < 60000) {
        auto unit = [&](double *v) {
            double n = 0;
            for (int i = 0; i < 3; ++i) v[i] = U() - 0.5, n += v[i] * v[i];
            n = std::sqrt(n);
            for (int i = 0; i < 3; ++i) v[i] /= n;
        };
        const double rho = std::ldexp(0.5 + 0.5 * U(), -(int)(8 * U()));
        const double D = rho * 2.0101 * std::pow(80.0, U() * U());
        double dir[3], off[3], nrm[3];
        unit(dir), unit(off), unit(nrm);
        const double f = U(), jw = 0.05 + 0.93 * U();
        const int e = float_exp((float)(D - rho)), eo = float_exp((float)rho);
        // the largest phases and dampings that the kernel takes, and less
        const double k = std::ldexp((U() < 0.5 ? -6.28 : 6.28) * (0.1 + 0.9 * U()), turns - e - (int)(4 * U()));
        double ki = 0.0;
        if (CPLX) {
            const double most = std::min(std::ldexp(0.69, kMaxDampExp - 1 - e), kMaxDampSpread / rho / 1.4427);
            ki = (U() < 0.5 ? -1 : 1) * most * std::pow(U(), 3) * 0.999;
        }
        if (ki == 0.0 && CPLX) continue;
        ++done;
        Pair P{};
        P.Dx = fixed((Q)dir[0] * D, 61 - e);
        P.Dy = fixed((Q)dir[1] * D, 61 - e);
        P.Dz = fixed((Q)dir[2] * D, 61 - e);
        P.osh = 1 + e - eo;
        int kx, kb, kdx = 0, kb2;
        const Q kt = frexpl((Q)k / (2 * pi), &kx);
        (void)frexpl((Q)k, &kb);
        if (CPLX) {
            (void)frexpl((Q)ki, &kb2);
            kb = std::max(kb, kb2) + 1;
        }
        pair_wavenumber(P, fixed(kt, 62), kx, fixed((Q)k, 62 - kb), kb, e);
        if (kx + e > kMaxTurnExp) return 1e9;
        if (CPLX) {
            const Q kd = frexpl((Q)ki * log2e, &kdx);
            if (kdx + e > kMaxDampExp) {
                --done;
                continue;
            }
            pair_damping(P, fixed(kd, 62), kdx, fixed((Q)ki, 62 - kb), kb, e,
                         pair_base((float)(ki * 1.4426950408889634), (float)D, (float)rho));
        }
        PointData g;
        Q d[3], r2 = 0, dn = 0;
        for (int i = 0; i < 3; ++i) {
            d[i] = (Q)dir[i] * D + (Q)off[i] * rho * f;
            r2 += d[i] * d[i];
            dn += d[i] * nrm[i];
        }
        g.ox = fixed((Q)off[0] * rho * f, 62 - eo);
        g.oy = fixed((Q)off[1] * rho * f, 62 - eo);
        g.oz = fixed((Q)off[2] * rho * f, 62 - eo);
        g.nx = split(fixed(nrm[0], 61));
        g.ny = split(fixed(nrm[1], 61));
        g.nz = split(fixed(nrm[2], 61));
        g.jw = split(fixed(jw, 63));
        const Point v = point<CPLX>(g, P, trig, damp);
        const Q r = sqrtl(r2), th = (Q)k * r, x = (Q)ki * r, t = dn * jw / (r2 * r), m = expl(-x);
        const Q c = cosl(th), s = sinl(th);
        const Q ref[4] = {m * (-(1 + x) * c - th * s) * t, m * (th * c - (1 + x) * s) * t, m * c * jw / r, m * s * jw / r};
        const int b = CPLX ? P.base : 0;
        const Q uF = ldexpl(1, -2 * e + P.fe - 58 - b), uG = ldexpl(1, -e - 58 - b);
        const Q got[4] = {v.Fr * uF, v.Fi * uF, v.Gr * uG, v.Gi * uG};
        // magnitudes over all phases and normals, the damping at the element's near end
        // (the values' unit, at most 2^5 above the point's own)
        const Q near = CPLX ? exp2l(-(Q)b) : 1, sf = near * jw / r2 * sqrtl((1 + fabsl(x)) * (1 + fabsl(x)) + th * th),
                sg = near * jw / r, size[4] = {sf, sf, sg, sg};
        for (int i = 0; i < 4; ++i) {
            const Q bound = 0x1p-50L + (fabsl(th) + fabsl(x)) * 0x1p-53L;
            worst = std::max(worst, (double)(fabsl(got[i] - ref[i]) / (size[i] * bound)));
        }
        if (CPLX && !(m <= near * 1.01L && m * 64 >= near)) return 1e9;
    }
    return worst;
}

int main(int argc, char **argv) {
    if (argc < 4) return 2;
    bool inside = true;
    const unsigned long long seed = (unsigned long long)std::atoll(argv[1]);
    const double worst = std::atoi(argv[3]) ? run<true>(seed, std::atoi(argv[2]), inside)
                                            : run<false>(seed, std::atoi(argv[2]), inside);
    std::printf("%d %.6f\n", inside ? 1 : 0, worst);
    return 0;
}
