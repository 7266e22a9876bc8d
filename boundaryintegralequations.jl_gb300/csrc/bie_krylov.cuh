// Pieces of the restarted GMRES kernels (bie_solver.cu, bie_cluster_gmres.cu):
// short complex vectors as components, sums over lanes, the small Hessenberg
// system.  A warp waits 62 cycles for each FP64 operation whatever its
// parallelism (measured), so what counts is the number of operations that a
// warp goes through: threads take real components, and serial recurrences
// spread over lanes.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace bie {
namespace krylov {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

// (a complex vector as components)
__device__ __forceinline__ const double *comps(const double2 *p) { return reinterpret_cast<const double *>(p); }
__device__ __forceinline__ double *comps(double2 *p) { return reinterpret_cast<double *>(p); }

// sum over groups of L neighbouring lanes (L a power of two up to 32)
__device__ __forceinline__ double lane_sum(double v, int L) {
    for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// lanes per component for ncol complex columns: T threads spread over them
template <int T>
__device__ __forceinline__ int lanes_per(int ncol) {
    int L = 32;
    while (L > 1 && L * 2 * ncol > T) L >>= 1;
    return L;
}

// Component im of conj(a) b added to s
__device__ __forceinline__ double dot_step(double s, double2 a, double2 b, bool im) {
    s = fma(a.x, im ? b.y : b.x, s);
    return fma(im ? -a.y : a.y, im ? b.x : b.y, s);
}
// Component im of a b added to s
__device__ __forceinline__ double mul_step(double s, double2 a, double2 b, bool im) {
    s = fma(a.x, im ? b.y : b.x, s);
    return fma(im ? a.y : -a.y, im ? b.x : b.y, s);
}

// Component `lane & 1` of (A x)[r] for a CSR row r (only where `in`), on eight
// neighbouring lanes: the two components times four shares of the row's
// non-zeros; every lane of a component gets the sum.  All lanes of the warp call
// it.  L2: x was written by other CTAs of this launch.
template <bool L2>
__device__ __forceinline__ double row_product(const int64_t *__restrict__ rp, const int32_t *__restrict__ cols,
                                              const double2 *__restrict__ val, const double2 *x, int64_t r, bool in,
                                              int lane) {
    const bool im = lane & 1;
    double v = 0.0;
    if (in) {
        const int64_t p1 = __ldg(rp + r + 1);
        for (int64_t p = __ldg(rp + r) + ((lane >> 1) & 3); p < p1; p += 16) {
            double2 c[4], b[4];   // (loads of four non-zeros in flight)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool ok = p + 4 * u < p1;
                const double2 *xp = x + (ok ? __ldg(cols + p + 4 * u) : 0);
                c[u] = ok ? __ldg(val + p + 4 * u) : make_double2(0.0, 0.0);
                b[u] = L2 ? __ldcg(xp) : *xp;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (p + 4 * u < p1) v = mul_step(v, c[u], b[u], im);
        }
    }
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v + __shfl_xor_sync(0xffffffffu, v, 4);
}

// The rotations 0 .. j-1 (cs real, sn complex) applied to col[0 .. j], by the
// first four lanes of a warp: lanes 0, 1 take the components of -conj(sn) a + c b,
// which the next rotation needs, lanes 2, 3 those of c a + sn b, the finished
// entry; three FP64 operations in a row for each rotation instead of twelve.
__device__ __forceinline__ void rotate_column(double2 *col, const double2 *sn, const double *cs, int j, int lane) {
    const bool im = lane & 1, fin = lane & 2;
    double2 a = col[0];
    __syncwarp(0xfu);   // lanes 2, 3 store col[0] in the first pass (the shuffles order the later entries)
    for (int k = 0; k < j; ++k) {
        const double2 b = col[k + 1], s = sn[k];
        const double2 p = fin ? a : b, q = fin ? b : a;
        double v = cs[k] * (im ? p.y : p.x);
        v = fma(fin ? s.x : -s.x, im ? q.y : q.x, v);
        v = fma(im ? s.y : -s.y, im ? q.x : q.y, v);
        if (fin) comps(col)[2 * k + im] = v;
        a = make_double2(__shfl_sync(0xfu, v, 0), __shfl_sync(0xfu, v, 1));
    }
    if (lane == 0) col[j] = a;
}

// The rotation that zeroes col[j + 1] = hn of (a, hn): cosine c, q = |sine|, sine
// sn and the new diagonal r, from na2 = |a|^2, ia = 1 / |a|, hn2 = hn^2, rh = 1 / hn
// and in = 1 / sqrt(na2 + hn2).  The squares are those of norms taken as roots
// of a sum of squares, so a scaled hypot would not widen the range.
struct Rotation {
    double c, q;
    double2 sn, r;
};
__device__ __forceinline__ Rotation last_rotation(double2 a, double na2, double ia, double hn2, double rh, double in) {
    if (hn2 == 0.0) return Rotation{1.0, 0.0, make_double2(0.0, 0.0), a};
    if (na2 == 0.0) return Rotation{0.0, 1.0, make_double2(1.0, 0.0), make_double2(hn2 * rh, 0.0)};
    const double q = hn2 * rh * in, t = q * ia, u = (na2 + hn2) * in * ia;
    return Rotation{na2 * ia * in, q, make_double2(a.x * t, a.y * t), make_double2(a.x * u, a.y * u)};
}

// y = R^{-1} y over j columns (back substitution by columns, one warp; ld > 0)
__device__ __forceinline__ void back_substitute(const double2 *R, int ld, int j, double2 *y, int lane) {
    for (int k = j - 1; k >= 0; --k) {
        const double2 d = R[(int64_t)k * ld + k];
        const double i = 1.0 / fma(d.x, d.x, d.y * d.y);
        const double2 yk = cmul(y[k], make_double2(d.x * i, -d.y * i));
        __syncwarp();
        if (lane == 0) y[k] = yk;
        for (int l = lane; l < k; l += 32) {
            const double2 t = cmul(R[(int64_t)k * ld + l], yk);
            y[l] = make_double2(y[l].x - t.x, y[l].y - t.y);
        }
        __syncwarp();
    }
}

}  // namespace krylov
}  // namespace bie
