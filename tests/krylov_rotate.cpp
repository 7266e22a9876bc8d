// Runs krylov::rotate_column (csrc/bie_krylov.cuh) on the host with one thread per
// lane, some of them late, against the rotations one after the other: prints the
// largest difference relative to the column.  Arguments: bit mask of the late
// lanes, rotations.
#include "bie_krylov.cuh"

#include <chrono>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <thread>
#include <vector>

int main(int argc, char **argv) {
    if (argc < 3) return 2;
    const int late = std::atoi(argv[1]), j = std::atoi(argv[2]);
    std::mt19937_64 gen(7);
    auto U = [&] { return (double)(gen() >> 11) * 0x1p-52 - 1.0; };
    std::vector<double2> col(j + 1), sn(j + 1);
    std::vector<double> cs(j + 1);
    std::vector<std::complex<double>> want;
    for (int k = 0; k <= j; ++k) {
        col[k] = make_double2(U(), U());
        want.push_back({col[k].x, col[k].y});
        const std::complex<double> s(U(), U());
        cs[k] = 1.0 / std::sqrt(1.0 + std::norm(s));
        sn[k] = make_double2(s.real() * cs[k], s.imag() * cs[k]);
    }
    for (int k = 0; k < j; ++k) {
        const std::complex<double> s(sn[k].x, sn[k].y), a = want[k], b = want[k + 1];
        want[k] = cs[k] * a + s * b;
        want[k + 1] = cs[k] * b - std::conj(s) * a;
    }
    std::vector<std::thread> lanes;
    for (int l = 0; l < host_warp::kLanes; ++l)
        lanes.emplace_back([&, l] {
            host_warp::lane = l;
            if ((late >> l) & 1) std::this_thread::sleep_for(std::chrono::milliseconds(100));
            bie::krylov::rotate_column(col.data(), sn.data(), cs.data(), j, l);
        });
    for (auto &t : lanes) t.join();
    double worst = 0, size = 0;
    for (int k = 0; k <= j; ++k) {
        worst = std::fmax(worst, std::abs(want[k] - std::complex<double>(col[k].x, col[k].y)));
        size = std::fmax(size, std::abs(want[k]));
    }
    std::printf("%g\n", worst / size);
    return 0;
}
