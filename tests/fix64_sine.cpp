// Drives the sine and cosine of bie_fixmath.cuh on the host against long double at
// one magnitude: prints the largest excess of the error over the final rounding, as
// a multiple of 2^-59, and the largest error of the sine in units in its last
// place.  Arguments: seed, binary exponent of the arguments.
#include "bie_fixmath.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace bie::fix64;
typedef long double Q;

int main(int argc, char **argv) {
    if (argc < 3) return 2;
    std::mt19937_64 gen((unsigned long long)std::atoll(argv[1]));
    const int e = std::atoi(argv[2]);
    auto U = [&] { return (double)(gen() >> 11) * 0x1p-53; };
    const Q pi = 3.141592653589793238462643383279502884L;
    static Limb tc[kTrigEntries], ts[kTrigEntries];
    for (int j = 0; j < kTrigEntries; ++j) {
        tc[j] = split((i64)llrintl(ldexpl(cosl(2 * pi * j / kTrigEntries), 62)));
        ts[j] = split((i64)llrintl(ldexpl(sinl(2 * pi * j / kTrigEntries), 62)));
    }
    auto trig = [&](int j, Limb &c, Limb &s) {
        c = tc[j];
        s = ts[j];
    };
    double excess = 0, ulp = 0;
    for (int n = 0; n < 200000; ++n) {
        const double x = (U() < 0.5 ? -1 : 1) * std::ldexp(1.0 + U(), e);
        double s, c;
        if (!sine_cosine<1076>(x, trig, s, c)) return 3;
        // reduced with 2 pi in two parts
        const Q hi = ldexpl((Q)0xc90fdaa22168c235ULL, -61), lo = -1.0033115225336664e-19L;
        const Q turns = rintl((Q)x / hi);
        const Q r = fmal(-turns, lo, fmal(-turns, hi, (Q)x));
        const Q want[2] = {sinl(r), cosl(r)};
        const double got[2] = {s, c};
        for (int k = 0; k < 2; ++k) {
            int q;
            (void)std::frexp((double)want[k], &q);
            const Q err = fabsl((Q)got[k] - want[k]);
            excess = std::fmax(excess, (double)((err - ldexpl(1.0L, q - 54)) / 0x1p-59L));
            if (k == 0) ulp = std::fmax(ulp, (double)(err / ldexpl(1.0L, q - 53)));
        }
    }
    std::printf("%.4f %.4f\n", excess, ulp);
    return 0;
}
