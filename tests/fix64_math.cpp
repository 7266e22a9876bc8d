// Drives the FP64 functions of bie_fixmath.cuh on the host against long double:
// prints the largest errors of 1 / sqrt, sqrt and e^-x in units in the last
// place and of sine and cosine as a multiple of their bound, then whether the
// arguments outside the ranges were refused.  Argument: a seed.
#include "bie_fixmath.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>

using namespace bie::fix64;
typedef long double Q;

static i64 fixed(Q x, int n) { return (i64)llrintl(ldexpl(x, n)); }
static double ulps(double x, Q y) {
    int e;
    (void)std::frexp((double)y, &e);
    return (double)(fabsl((Q)x - y) / ldexpl(1.0L, e - 53));
}

int main(int argc, char **argv) {
    if (argc < 2) return 2;
    std::mt19937_64 gen((unsigned long long)std::atoll(argv[1]));
    auto U = [&] { return (double)(gen() >> 11) * 0x1p-53; };
    const Q pi = 3.141592653589793238462643383279502884L;
    static Limb tc[kTrigEntries], ts[kTrigEntries], td[kDampEntries];
    for (int j = 0; j < kTrigEntries; ++j) {
        tc[j] = split(fixed(cosl(2 * pi * j / kTrigEntries), 62));
        ts[j] = split(fixed(sinl(2 * pi * j / kTrigEntries), 62));
    }
    for (int j = 0; j < kDampEntries; ++j) td[j] = split(fixed(exp2l(-(Q)j / kDampEntries), 62));
    bool ok = true;
    auto trig = [&](int j, Limb &c, Limb &s) {
        ok = ok && j >= 0 && j < kTrigEntries;
        c = tc[j & (kTrigEntries - 1)];
        s = ts[j & (kTrigEntries - 1)];
    };
    auto damp = [&](int j) {
        ok = ok && j >= 0 && j < kDampEntries;
        return td[j & (kDampEntries - 1)];
    };
    double er = 0, es = 0, ee = 0, et = 0;
    for (int n = 0; n < 200000; ++n) {
        const double x2 = std::ldexp(1.0 + U(), (int)(1990 * U()) - 995);
        double ri, r, v, s, c;
        ok = ok && root(x2, ri, r);
        er = std::fmax(er, ulps(ri, 1 / sqrtl((Q)x2)));
        es = std::fmax(es, ulps(r, sqrtl((Q)x2)));
        const double y = (U() < 0.3 ? -1 : 1) * std::pow(10.0, 14 * U() - 12) * 6.9;
        if (std::fabs(y) < 700.0) {
            ok = ok && exp_minus(y, damp, v);
            ee = std::fmax(ee, ulps(v, expl(-(Q)y)));
        }
        const double x = (U() < 0.5 ? -1 : 1) * std::ldexp(1.0 + U(), (int)(79 * U()) - 60);
        ok = ok && sine_cosine(x, trig, s, c);
        const Q bound = ldexpl(1.0L, -59) + fabsl((Q)x) * ldexpl(1.0L, -61);
        for (int k = 0; k < 2; ++k) {
            const double got = k ? c : s;
            const Q want = k ? cosl((Q)x) : sinl((Q)x);
            int e;
            (void)std::frexp(got, &e);
            et = std::fmax(et, (double)(fabsl((Q)got - want) / (bound + ldexpl(1.0L, e - 54))));
        }
    }
    double a, b;
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    for (double x : {0.0, -1.0, inf, -inf, nan, 1e-305, 1e305}) ok = ok && !root(x, a, b);
    for (double x : {inf, -inf, nan, 1e7, -1e300}) ok = ok && !sine_cosine(x, trig, a, b);
    for (double x : {inf, -inf, nan, 700.0, -700.0}) ok = ok && !exp_minus(x, damp, a);
    ok = ok && sine_cosine(0.0, trig, a, b) && std::fabs(a) < 0x1p-59 && std::fabs(b - 1.0) < 0x1p-52;
    ok = ok && sine_cosine(5e-324, trig, a, b) && std::fabs(a) < 0x1p-59;
    ok = ok && exp_minus(0.0, damp, a) && a == 1.0;
    std::printf("%g %g %g %g %d\n", er, es, ee, et, ok ? 1 : 0);
    return 0;
}
