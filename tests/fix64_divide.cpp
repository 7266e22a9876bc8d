// Drives the division, square root and hypot of bie_fixmath.cuh on the host
// against the IEEE operations: prints how many results differ in any bit.
// Argument: a seed.  (Compiled without FMA contraction.)
#include "bie_fixmath.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace bie::fix64;

static double julia_hypot(double x, double y, double z) {
    const double m = std::fmax(std::fmax(std::fabs(x), std::fabs(y)), std::fabs(z));
    const double a = x / m, b = y / m, c = z / m;
    return m * std::sqrt((a * a + b * b) + c * c);
}

int main(int argc, char **argv) {
    if (argc < 2) return 2;
    std::mt19937_64 gen((unsigned long long)std::atoll(argv[1]));
    auto U = [&] { return (double)(gen() >> 11) * 0x1p-53; };
    auto any = [&](int range) { return (U() < 0.5 ? -1 : 1) * std::ldexp(1 + U(), (int)(2 * range * U()) - range); };
    long div = 0, root = 0, hyp = 0, refused = 0;
    for (int n = 0; n < 500000; ++n) {
        double b = std::fabs(any(20)), a = any(20);
        if (n % 5 == 0) a = (int)(1 + U() * 1000), b = (int)(1 + U() * 1000);   // exact and short quotients
        if (n % 7 == 0) a = b * (1 + (int)(U() * 8 - 4) * 0x1p-52);             // quotients next to one
        if (n % 11 == 0) b = std::ldexp(1.0, (int)(U() * 20));                  // powers of two
        if (n % 13 == 0) a = -0.0;
        const double q = divide(a, divisor(b));
        div += double_bits(q) != double_bits(a / b);
        double x = 1 + 3 * U();
        if (n % 3 == 0) x = std::pow(1 + (int)(U() * 300) / 300.0, 2);          // squares
        if (x < 4) root += square_root(x) != std::sqrt(x);
        const double u = any(15), v = n % 4 ? any(15) : 0.0, w = n % 9 ? any(15) : -u;
        double h = 0;
        if (!hypot3(u, v, w, h)) ++refused;
        else hyp += h != julia_hypot(u, v, w);
    }
    double h;
    bool edges = !hypot3(0, 0, 0, h) && !hypot3(1.0, 1e-40, 0, h) && !hypot3(1e300, 0, 0, h) &&
                 !hypot3(1e-300, 1e-300, 0, h) && !hypot3(INFINITY, 1, 1, h) && !hypot3(NAN, 1, 1, h) &&
                 hypot3(0, 3, 4, h) && h == 5.0;
    std::printf("%ld %ld %ld %ld %d\n", div, root, hyp, refused, edges ? 1 : 0);
    return 0;
}
