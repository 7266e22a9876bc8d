// Drives the element factors of bie_fix64.cuh on the host against long double:
// prints the largest error of value times factor in units of the value's last
// place over factors of all magnitudes, then whether zero and the exponents are
// as they should be.  Argument: a seed.
#include "bie_fix64.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace bie::fix64;
typedef long double Q;

int main(int argc, char **argv) {
    if (argc < 2) return 2;
    std::mt19937_64 gen((unsigned long long)std::atoll(argv[1]));
    auto U = [&] { return (double)(gen() >> 11) * 0x1p-53; };
    double worst = 0;
    bool ok = true;
    for (int n = 0; n < 200000; ++n) {
        const int s = (int)(800 * U()) - 400, t = (int)(60 * U());
        double re = std::ldexp(2 * U() - 1, s), im = std::ldexp(2 * U() - 1, s - t);
        if (n % 7 == 0) std::swap(re, im);
        if (n % 11 == 0) im = 0;
        const Factor f = element_factor(re, im);
        const double top = std::fmax(std::fabs(re), std::fabs(im));
        ok = ok && top >= std::ldexp(0.5, f.e) && top < std::ldexp(1.0, f.e);
        const i64 a = (i64)llrintl(ldexpl(2 * U() - 1, 59)), b = (i64)llrintl(ldexpl(2 * U() - 1, 59));
        const Values2 v = complex_mul(split(a), split(b), f.re, f.im);
        const Q fr = ldexpl((Q)re, -f.e), fi = ldexpl((Q)im, -f.e);
        worst = std::fmax(worst, (double)fabsl((Q)v.re - ((Q)a * fr - (Q)b * fi)));
        worst = std::fmax(worst, (double)fabsl((Q)v.im - ((Q)a * fi + (Q)b * fr)));
    }
    const Factor z = element_factor(0.0, -0.0);
    ok = ok && z.e == kZeroFactor && z.re.h == 0 && z.re.l == 0 && z.im.h == 0 && z.im.l == 0;
    std::printf("%.3f %d\n", worst, ok ? 1 : 0);
    return 0;
}
