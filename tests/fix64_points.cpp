// Drives the fixed-point quadrature points of bie_fix64.cuh on the host against
// long double: prints the largest error of F, G and t over random regular pairs
// as a multiple of its bound.  Argument: a seed.
#include "bie_fix64.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace bie::fix64;
typedef long double Q;

static i64 fixed(Q x, int n) { return (i64)llrintl(ldexpl(x, n)); }

int main(int argc, char **argv) {
    if (argc < 2) return 2;
    std::mt19937_64 gen((unsigned long long)std::atoll(argv[1]));
    auto U = [&] { return (double)(gen() >> 11) * 0x1p-53; };
    const Q pi = 3.141592653589793238462643383279502884L;
    static Limb tc[kTrigEntries], ts[kTrigEntries];
    for (int j = 0; j < kTrigEntries; ++j) {
        tc[j] = split(fixed(cosl(2 * pi * j / kTrigEntries), 62));
        ts[j] = split(fixed(sinl(2 * pi * j / kTrigEntries), 62));
    }
    bool inside = true;
    auto trig = [&](int j, Limb &c, Limb &s) {
        inside = inside && j >= 0 && j < kTrigEntries;
        c = tc[j & (kTrigEntries - 1)];
        s = ts[j & (kTrigEntries - 1)];
    };
    auto damp = [](int) { return Limb{0, 0}; };   // complex k only
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
        const double D = rho * 2.0101 * std::pow(80.0, U() * U());   // |D| >= 2.01 rho
        double dir[3], off[3], nrm[3];
        unit(dir), unit(off), unit(nrm);
        const double f = U(), jw = 0.05 + 0.93 * U(), k = std::pow(10.0, 4 * U() - 2) * (U() < 0.5 ? -1 : 1);
        const int e = float_exp((float)(D - rho)), eo = float_exp((float)rho);
        if (std::fabs(k) * std::ldexp(1.0, e) / 6.2832 >= 512.0) continue;
        ++done;
        Pair P{};
        P.Dx = fixed((Q)dir[0] * D, 61 - e);
        P.Dy = fixed((Q)dir[1] * D, 61 - e);
        P.Dz = fixed((Q)dir[2] * D, 61 - e);
        P.osh = 1 + e - eo;
        int kx, kb;
        const Q kt = frexpl((Q)k / (2 * pi), &kx), km = frexpl((Q)k, &kb);
        pair_wavenumber(P, fixed(kt, 62), kx, fixed(km, 62), kb, e);
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
        const Point v = point<false>(g, P, trig, damp);
        const Q r = sqrtl(r2), th = (Q)k * r, t = dn * jw / (r2 * r);
        const Q c = cosl(th), s = sinl(th);
        const Q ref[5] = {(-c - s * th) * t, (c * th - s) * t, c * jw / r, s * jw / r, t};
        const Q uF = ldexpl(1, -2 * e + P.fe - 58), uG = ldexpl(1, -e - 58), uT = ldexpl(1, -2 * e - 57);
        const Q got[5] = {v.Fr * uF, v.Fi * uF, v.Gr * uG, v.Gi * uG, v.tq * uT};
        // magnitudes of the values over all phases and normals; bound: 2^-50 for
        // the roundings (a few units of 2^-58 .. 2^-57 of values that are at least
        // 0.05 / 9 of their range) and 2^-53 of the phase (r to 2^-55, the table)
        const Q sf = jw / r2 * sqrtl(1 + th * th), size[5] = {sf, sf, jw / r, jw / r, jw / r2};
        for (int i = 0; i < 5; ++i) {
            const Q bound = 0x1p-50L + (i < 4 ? fabsl(th) * 0x1p-53L : 0);
            worst = std::max(worst, (double)(fabsl(got[i] - ref[i]) / (size[i] * bound)));
        }
    }
    std::printf("%d %.6f\n", inside ? 1 : 0, worst);
    return 0;
}
