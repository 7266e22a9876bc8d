// Stand-ins for the CUDA names that csrc/bie_krylov.cuh uses, so that its warp
// code runs on the host: one thread per lane, and a barrier of the lanes behind
// every warp operation.
#pragma once

#include <barrier>
#include <cmath>
#include <cstdint>

#define __device__
#define __forceinline__ inline

struct double2 {
    double x, y;
};
inline double2 make_double2(double x, double y) { return double2{x, y}; }
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }
using std::fma;
template <class T>
T __ldg(const T *p) { return *p; }
template <class T>
T __ldcg(const T *p) { return *p; }

namespace host_warp {
constexpr int kLanes = 4;
inline std::barrier<> gate(kLanes);
inline double slots[kLanes];
inline thread_local int lane = 0;
}  // namespace host_warp
inline double __shfl_sync(unsigned, double v, int from) {
    host_warp::slots[host_warp::lane] = v;
    host_warp::gate.arrive_and_wait();
    const double r = host_warp::slots[from];
    host_warp::gate.arrive_and_wait();
    return r;
}
inline double __shfl_xor_sync(unsigned m, double v, int o) { return __shfl_sync(m, v, host_warp::lane ^ o); }
inline void __syncwarp(unsigned = 0xffffffffu) { host_warp::gate.arrive_and_wait(); }
