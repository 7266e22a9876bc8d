// K7: adjoint gradient of a far-field objective with respect to vertex
// positions and per-element boundary impedance (bie_adjoint).
//
// Forward model (3-node triangles with nodal physics on the vertices, the
// configuration of the shape/impedance study):
//   A p = p_I,   A = F + Diagonal(1 - C) - i rho c k G_Y,
//   G_Y[i, a] = sum_e Y_e G^(e)[i, a],  Y_e = 1 / Z_e  (element admittance),
// i.e. the boundary integral equation of README.md:10-18 with the impedance
// condition v_n = p / Z on each element, F, G, C as assembled by
// assemble_parallel! (src/3d/assembly_collocation.jl:270-353) and the
// exterior collocation form of test/3d/assembly_test.jl:37.  The reference's
// closest impedance form is nodal (examples/3d_cube_wave_anechoic.jl:62-68);
// the per-element admittance is defined here.
//   p_f = p_I(x_f) + B p,   B = -F_x + i rho c k G_{x,Y}   (field points x_f),
//   J = sum_j |p_f(x_j)|^2,  p_I(x) = exp(-i k d.x)  (incoming_wave,
//   src/analytical/3d_scattering.jl:4-12).
// Adjoint: A^H lambda = B^H p_f, then
//   dJ = 2 Re[ p_f^H dB p - lambda^H dA p + lambda^H dp_I ].
// The reverse pass recomputes the quadrature of every (row, element) pair
// with the forward rule choice (the nearest-node rule is piecewise constant
// in the geometry) and accumulates analytic derivatives of the integrands
// with respect to the element vertices, the collocation point and Y_e: in FP64
// for BIE_PREC_FP64 (adjoint_grad_kernel), in double-float with the near pairs in
// FP64 for BIE_PREC_DF64 (adjoint_df64_kernel).
#include "bie_internal.h"
#include "bie_device.cuh"
#include "bie_df64.cuh"
#include "bie_fixmath.cuh"

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

namespace bie {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr int kT = 128;

struct cd {
    double re, im;
};
__device__ __forceinline__ cd cmul(cd a, cd b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ cd cadd(cd a, cd b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ cd cscale(cd a, double s) { return {a.re * s, a.im * s}; }
__device__ __forceinline__ cd cconj(cd a) { return {a.re, -a.im}; }

// ---------------------------------------------------------------------------
// small kernels of the driver
// ---------------------------------------------------------------------------
__global__ void admittance_kernel(const double2 *__restrict__ Z, const int32_t *__restrict__ order,
                                  int64_t E, double2 *__restrict__ Y) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= E) return;
    const double2 z = Z[order[p]];
    const double den = z.x * z.x + z.y * z.y;
    Y[p] = make_double2(z.x / den, -z.y / den);
}

// A = F + a G (in place in F), A_ii += 1 - C_i  (diag only when C != null)
__global__ void combine_system_kernel(double2 *__restrict__ F, const double2 *__restrict__ G,
                                      double2 a, const double2 *__restrict__ C, int64_t M,
                                      int64_t N) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < M * N; t += stride) {
        const double2 f = F[t], g = G[t];
        double re = f.x + a.x * g.x - a.y * g.y, im = f.y + a.x * g.y + a.y * g.x;
        if (C) {
            const int64_t i = t % M, j = t / M;
            if (i == j) {
                re += 1.0 - C[i].x;
                im += -C[i].y;
            }
        }
        F[t] = make_double2(re, im);
    }
}

// p_I(x) = exp(-i k d.x) at n points (3 x n)
__global__ void incident_kernel(const double *__restrict__ X, int64_t n, double kre, double kim,
                                double dx, double dy, double dz, double2 *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double s = dx * X[3 * i] + dy * X[3 * i + 1] + dz * X[3 * i + 2];
    // -i k s = kim s - i kre s
    const double mag = exp(kim * s);
    double sn, cs;
    sincos(-kre * s, &sn, &cs);
    out[i] = make_double2(mag * cs, mag * sn);
}

// y[i] = b0[i] + sum_j B[i + j M] p[j]   (M small), one warp per row
__global__ void small_gemv_kernel(const double2 *__restrict__ B, int64_t M, int64_t N,
                                  const double2 *__restrict__ p, const double2 *__restrict__ b0,
                                  double2 *__restrict__ y) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= M) return;
    double re = 0, im = 0;
    for (int64_t j = lane; j < N; j += 32) {
        const double2 b = B[row + j * M], v = p[j];
        re += b.x * v.x - b.y * v.y;
        im += b.x * v.y + b.y * v.x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (lane == 0) y[row] = make_double2(b0[row].x + re, b0[row].y + im);
}

// r[j] = sum_i conj(B[i + j M]) pf[i]   (B^H pf), one thread per column
__global__ void adjoint_rhs_kernel(const double2 *__restrict__ B, int64_t M, int64_t N,
                                   const double2 *__restrict__ pf, double2 *__restrict__ r) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N) return;
    double re = 0, im = 0;
    for (int64_t i = 0; i < M; ++i) {
        const double2 b = B[i + j * M], v = pf[i];
        re += b.x * v.x + b.y * v.y;
        im += b.x * v.y - b.y * v.x;
    }
    r[j] = make_double2(re, im);
}

// At = A^H (N x N column-major), 32 x 32 tiles through shared memory
__global__ void conj_transpose_kernel(const double2 *__restrict__ A, double2 *__restrict__ At, int64_t N) {
    __shared__ double2 tile[32][33];
    const int64_t bx = (int64_t)blockIdx.x * 32, by = (int64_t)blockIdx.y * 32;
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const int64_t i = bx + threadIdx.x, j = by + yy;   // A[i, j]
        if (i < N && j < N) tile[yy][threadIdx.x] = A[i + j * N];
    }
    __syncthreads();
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const int64_t i = by + threadIdx.x, j = bx + yy;   // At[i, j] = conj(A[j, i])
        if (i < N && j < N) {
            const double2 v = tile[threadIdx.x][yy];
            At[i + j * N] = make_double2(v.x, -v.y);
        }
    }
}

// ---------------------------------------------------------------------------
// Reverse pass.  Rows: [0, N) collocation rows of A (target = node i, weight
// w_i = -lambda_i, alpha_F = 1, alpha_G = -i rho c k, C term), [N, N + M)
// field rows of B (weight p_f, alpha_F = -1, alpha_G = +i rho c k).
// For L = Re sum_rows conj(w) [row . p] the kernel accumulates dL/dX for the
// vertices (atomics), and s_e = dL_complex/dY_e per element.
// ---------------------------------------------------------------------------
struct RuleTab {
    int Q[3];
    int off[3];   // first point of rule r in the table (4 doubles per point: N1 N2 N3 w)
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <bool CPLX_K>
__global__ void __launch_bounds__(kT)
adjoint_grad_kernel(int64_t N, int64_t M, const double *__restrict__ src, const double *__restrict__ fpts,
                    const double2 *__restrict__ w, const double2 *__restrict__ p,
                    const double *__restrict__ coords, const int32_t *__restrict__ topo,
                    const int32_t *__restrict__ order, const double2 *__restrict__ Y, int64_t E, int S,
                    const double *__restrict__ tab, RuleTab rt, const int32_t *__restrict__ trig_tab, double kre,
                    double kim, double rhock, double *__restrict__ dX, double2 *__restrict__ sY) {
    const dev::TrigFix trig{trig_tab};
    const int64_t row = (int64_t)blockIdx.x * kT + threadIdx.x;
    const bool active = row < N + M;
    const bool arow = row < N;
    const int s = blockIdx.y;
    const int64_t e0 = (int64_t)s * E / S, e1 = (int64_t)(s + 1) * E / S;
    double tx = 0, ty = 0, tz = 0;
    cd cw = {0, 0}, pi = {0, 0};
    if (active) {
        const double *T = arow ? src + 3 * row : fpts + 3 * (row - N);
        tx = T[0];
        ty = T[1];
        tz = T[2];
        const double2 wv = w[row];
        cw = {wv.x, -wv.y};   // conj(w)
        if (arow) pi = {p[row].x, p[row].y};
    }
    // alpha_F, alpha_G per row kind
    const double aF = arow ? 1.0 : -1.0;
    const cd aG = arow ? cd{0.0, -rhock} : cd{0.0, rhock};
    const cd ik = {-kim, kre};
    const double inv4pi = 1.0 / (4.0 * kPi);
    double gtx = 0, gty = 0, gtz = 0;   // d L / d target (collocation node)

    for (int64_t pe = e0; pe < e1; ++pe) {
        const int64_t e = order[pe];
        const int32_t n0 = topo[3 * e], n1 = topo[3 * e + 1], n2 = topo[3 * e + 2];
        double X[9];
        X[0] = coords[3 * n0]; X[1] = coords[3 * n0 + 1]; X[2] = coords[3 * n0 + 2];
        X[3] = coords[3 * n1]; X[4] = coords[3 * n1 + 1]; X[5] = coords[3 * n1 + 2];
        X[6] = coords[3 * n2]; X[7] = coords[3 * n2 + 1]; X[8] = coords[3 * n2 + 2];
        const double2 yv = Y[pe];
        const cd Ye = {yv.x, yv.y};
        const cd p0 = {p[n0].x, p[n0].y}, p1 = {p[n1].x, p[n1].y}, p2 = {p[n2].x, p[n2].y};
        // element vectors
        const double ux = X[3] - X[0], uy = X[4] - X[1], uz = X[5] - X[2];
        const double vx = X[6] - X[0], vy = X[7] - X[1], vz = X[8] - X[2];
        const double nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
        const double jac = sqrt(nx * nx + ny * ny + nz * nz);
        double g1x = 0, g1y = 0, g1z = 0, g2x = 0, g2y = 0, g2z = 0, g3x = 0, g3y = 0, g3z = 0;
        double Gnx = 0, Gny = 0, Gnz = 0;
        cd se = {0, 0};
        if (active) {
            const int c = dev::nearest_node<3>(X, tx, ty, tz);
            const double *P = tab + 4 * (int64_t)rt.off[c];
            const int Q = rt.Q[c];
            for (int q = 0; q < Q; ++q) {
                const double N1 = P[4 * q], N2 = P[4 * q + 1], N3 = P[4 * q + 2], wq = P[4 * q + 3];
                const double yx = N1 * X[0] + N2 * X[3] + N3 * X[6];
                const double yy = N1 * X[1] + N2 * X[4] + N3 * X[7];
                const double yz = N1 * X[2] + N2 * X[5] + N3 * X[8];
                const double dx = yx - tx, dy = yy - ty, dz = yz - tz;
                const double r2 = dx * dx + dy * dy + dz * dz;
                double rinv, r, sn, cs;
                trig.root_of(r2, rinv, r);
                trig.sincos_of(kre * r, &sn, &cs);
                if (CPLX_K) {
                    const double dmp = trig.exp_minus(kim * r);
                    sn *= dmp;
                    cs *= dmp;
                }
                const cd E1 = {cs, sn};                       // e^{ikr}
                const cd ikr = cscale(ik, r);
                const cd ikr1 = {ikr.re - 1.0, ikr.im};
                const double ri2 = rinv * rinv, ri3 = ri2 * rinv, ri4 = ri2 * ri2;
                // phi_F = -e^{ikr}(ikr-1)/(4 pi r^3), phi_F' = e^{ikr}(k^2/r^2 + 3(ikr-1)/r^4)/(4 pi)
                const cd phiF = cscale(cmul(E1, ikr1), -inv4pi * ri3);
                const cd k2 = cmul(ik, ik);                   // (ik)^2 = -k^2
                const cd dphiF = cscale(cmul(E1, cadd(cscale(k2, -ri2), cscale(ikr1, 3.0 * ri4))), inv4pi);
                // phi_G = e^{ikr}/(4 pi r), phi_G' = e^{ikr}(ikr - 1)/(4 pi r^2)
                const cd phiG = cscale(E1, inv4pi * rinv);
                const cd dphiG = cscale(cmul(E1, ikr1), inv4pi * ri2);
                // phi_C = -1/(4 pi r^3), phi_C' = 3/(4 pi r^4)
                const double phiC = -inv4pi * ri3, dphiC = 3.0 * inv4pi * ri4;
                const cd Ph = cadd(cadd(cscale(p0, N1), cscale(p1, N2)), cscale(p2, N3));
                const cd base = cscale(cmul(cw, Ph), wq);     // conj(w) Ph w_q
                const cd SF = cscale(base, aF);
                const cd SG = cmul(cmul(base, aG), Ye);
                const cd SC = arow ? cscale(cmul(cw, pi), wq) : cd{0, 0};
                const double dn = dx * nx + dy * ny + dz * nz;
                const double coef_r = cmul(SF, dphiF).re * dn + cmul(SG, dphiG).re * jac + SC.re * dphiC * dn;
                const double coef_n = cmul(SF, phiF).re + SC.re * phiC;
                const double coef_j = cmul(SG, phiG).re / jac;
                const double gdx = coef_r * dx * rinv + coef_n * nx;
                const double gdy = coef_r * dy * rinv + coef_n * ny;
                const double gdz = coef_r * dz * rinv + coef_n * nz;
                Gnx += coef_n * dx + coef_j * nx;
                Gny += coef_n * dy + coef_j * ny;
                Gnz += coef_n * dz + coef_j * nz;
                g1x += N1 * gdx; g1y += N1 * gdy; g1z += N1 * gdz;
                g2x += N2 * gdx; g2y += N2 * gdy; g2z += N2 * gdz;
                g3x += N3 * gdx; g3y += N3 * gdy; g3z += N3 * gdz;
                gtx -= gdx; gty -= gdy; gtz -= gdz;
                se = cadd(se, cmul(cmul(base, aG), cscale(phiG, jac)));
            }
            // nn = u x v: dL/du = v x Gn, dL/dv = Gn x u
            const double aux = vy * Gnz - vz * Gny, auy = vz * Gnx - vx * Gnz, auz = vx * Gny - vy * Gnx;
            const double avx = Gny * uz - Gnz * uy, avy = Gnz * ux - Gnx * uz, avz = Gnx * uy - Gny * ux;
            g2x += aux; g2y += auy; g2z += auz;
            g3x += avx; g3y += avy; g3z += avz;
            g1x -= aux + avx; g1y -= auy + avy; g1z -= auz + avz;
        }
        // reduce over the warp's rows, one set of atomics per warp and element
        g1x = warp_sum(g1x); g1y = warp_sum(g1y); g1z = warp_sum(g1z);
        g2x = warp_sum(g2x); g2y = warp_sum(g2y); g2z = warp_sum(g2z);
        g3x = warp_sum(g3x); g3y = warp_sum(g3y); g3z = warp_sum(g3z);
        se.re = warp_sum(se.re);
        se.im = warp_sum(se.im);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&dX[3 * n0], g1x); atomicAdd(&dX[3 * n0 + 1], g1y); atomicAdd(&dX[3 * n0 + 2], g1z);
            atomicAdd(&dX[3 * n1], g2x); atomicAdd(&dX[3 * n1 + 1], g2y); atomicAdd(&dX[3 * n1 + 2], g2z);
            atomicAdd(&dX[3 * n2], g3x); atomicAdd(&dX[3 * n2 + 1], g3y); atomicAdd(&dX[3 * n2 + 2], g3z);
            atomicAdd(&sY[e].x, se.re);
            atomicAdd(&sY[e].y, se.im);
        }
    }
    if (active && arow) {   // the collocation point is vertex `row`
        atomicAdd(&dX[3 * row], gtx);
        atomicAdd(&dX[3 * row + 1], gty);
        atomicAdd(&dX[3 * row + 2], gtz);
    }
}

// ---------------------------------------------------------------------------
// The reverse pass on the FP32 pipes (BIE_PREC_DF64).
//
// adjoint_grad_kernel is bound by the FP64 pipe (87 % busy, 67 ms for the
// 4842-node ellipsoid, 46.9 M pairs).  Here the regular pairs run in double-float
// (bie_df64.cuh) and only near pairs and nearest-node near-ties in FP64, in place:
// 13.0 ms, bound by instruction issue and half by instruction fetch (128
// registers, 16 warps per SM; two rows per thread with one reduction for both took
// 19.7 ms at 255 registers): the loop over elements is longer than the
// instruction caches, so the warps of a block stay together.  Whole gradient 28.2
// ms without that, 26.9 in blocks of 128 threads, 25.8 of 256, 27.4 of 512.  Phases
// are formed without cancellation.  Error of a gradient with the solves carried on
// to 3e-16 (a tolerance of 1e-13 leaves 1e-13 .. 9e-13), ellipsoids of 252 to 2562
// nodes at k = 3, field points at 10: 2e-14 .. 4e-14, with the FP64 kernel 3e-15 ..
// 1e-14; at k = 0.3 or with field points at 1.5 it is 5e-15 .. 5e-14 against 1e-15 ..
// 6e-15, so FP64 callers keep the FP64 kernel.  With
// b = conj(w) p(x_q), z = b e^{ikr}, W = jw / 4 pi, n the unit normal, d = x_q - t,
// g = z alpha_G Y_e, sc = Re conj(w) p_i (collocation rows):
//   t3 = alpha_F (z_r + k r z_i) - sc,     gp = Re g (i k r - 1),
//   A' = W/r^2 [ (d.n)/r (alpha_F k^2 z_r - 3 t3 / r^2) + gp / r ],  B = W t3 / r^3,
//   dL/dx_q = A' d + B n,   dL/dnn = (B d + W g_r / r n) / J   (nn = u x v = J n).
// Since x_q = sum_a N_a X_a, a pair needs only the scalars
//   M_ab = sum_q A' N_a N_b,  SB_a = sum_q B N_a,  SG = sum_q W g_r / r,
//   SZ = sum_q z W / r,
// and over all rows an element needs the sums of M_ab, D M_a, SB_a, D SB, SG, SZ
// (M_a = sum_b M_ab, D = centroid - t): 24 numbers, reduced over a warp's rows
// and added to the element's accumulators; adjoint_finish_kernel forms the vertex
// gradients from them once per element in FP64.
// ---------------------------------------------------------------------------
using dev::df;
using df64::dd::Acc;
namespace dd = df64::dd;
constexpr int kAdjSums = 24;       // M 0..5, D M_a 6..14, SB_a 15..17, D SB 18..20, SG 21, SZ 22, 23
constexpr int kAdjTab = 20;        // floats per rule point: N_a N_b (11 22 33 12 13 23), N_a as hi, lo

struct AdjPair {                   // the scalars of one pair
    double M[6], SB[3], SG, SZr, SZi;
};

struct AdjView {
    const double *rec;             // FP64 records
    int stride, nidx_off, qmax;
    const double *phi;
    const int32_t *tab;            // tables of dev::TrigFix
    dev::RuleInfo ri;
};

// One pair in FP64 (near pairs: the reference's rule choice and arithmetic).
__device__ __noinline__ AdjPair adjoint_pair_fp64(const AdjView &v, int64_t pe, double tx, double ty, double tz,
                                                  cd cw, double sc, double aF, double sgn, cd G0,
                                                  const double2 *__restrict__ p, double kre) {
    const double *r = v.rec + (size_t)pe * v.stride;
    const int c = dev::nearest_node<3>(r, tx, ty, tz);
    const int Q = v.ri.Q[c];
    const dev::TrigFix trig{v.tab};
    const double *g = r + v.ri.off[c], *ph = v.phi + (size_t)c * v.qmax * 3;
    const int32_t *nid = reinterpret_cast<const int32_t *>(r + v.nidx_off);
    const cd p0 = {p[nid[0]].x, p[nid[0]].y}, p1 = {p[nid[1]].x, p[nid[1]].y}, p2 = {p[nid[2]].x, p[nid[2]].y};
    AdjPair o;
    for (int j = 0; j < 6; ++j) o.M[j] = 0.0;
    for (int j = 0; j < 3; ++j) o.SB[j] = 0.0;
    o.SG = o.SZr = o.SZi = 0.0;
    for (int q = 0; q < Q; ++q) {
        const double N1 = ph[3 * q], N2 = ph[3 * q + 1], N3 = ph[3 * q + 2];
        const double dx = g[q] - tx, dy = g[Q + q] - ty, dz = g[2 * Q + q] - tz;
        const double r2 = dx * dx + dy * dy + dz * dz;
        double ri, rr, sn, cs;
        trig.root_of(r2, ri, rr);
        const double ri2 = ri * ri;
        trig.sincos_of(kre * rr, &sn, &cs);
        const cd Ph = cadd(cadd(cscale(p0, N1), cscale(p1, N2)), cscale(p2, N3));
        const cd z = cmul(cmul(cw, Ph), cd{cs, sn});
        const double kr = kre * rr;
        const double t3 = aF * (z.re + kr * z.im) - sc;
        const cd gg = cmul(z, G0);
        const double gp = -sgn * (gg.re + kr * gg.im);
        const double wr = g[6 * Q + q] * dev::kInv4Pi * ri;
        // (d.n)/r with the outward normal: the record holds its negative
        const double dh = -(g[3 * Q + q] * dx + g[4 * Q + q] * dy + g[5 * Q + q] * dz) * ri;
        const double A = wr * ri * (dh * (aF * kre * kre * z.re - 3.0 * t3 * ri2) + gp * ri);
        const double B = wr * ri2 * t3;
        o.M[0] += A * N1 * N1;
        o.M[1] += A * N2 * N2;
        o.M[2] += A * N3 * N3;
        o.M[3] += A * N1 * N2;
        o.M[4] += A * N1 * N3;
        o.M[5] += A * N2 * N3;
        o.SB[0] += B * N1;
        o.SB[1] += B * N2;
        o.SB[2] += B * N3;
        o.SG += wr * sgn * gg.re;
        o.SZr += wr * sgn * z.re;
        o.SZi += wr * sgn * z.im;
    }
    return o;
}

// (K + k3) a with k3 the third float of the wavenumber: a wavenumber rounded to
// 48 bits is a systematic relative error, which the sums over rows and elements do
// not average (gradient error 2.4e-13 without it, 1e-13 from the solves alone)
__device__ __forceinline__ df mul_k(df K, float k3, df a) {
    const float p = __fmul_rn(K.hi, a.hi);
    float e = __fmaf_rn(K.hi, a.hi, -p);
    e = __fmaf_rn(K.hi, a.lo, e);
    e = __fmaf_rn(K.lo, a.hi, e);
    return dev::fast_two_sum(p, __fmaf_rn(k3, a.hi, e));
}
__device__ __forceinline__ float third(double x, df a) {
    return (float)((x - (double)a.hi) - (double)a.lo);
}
__device__ __forceinline__ void acc_prod(Acc &s, df a, df b) { dd::acc_add(s, dd::mul_raw(a, b)); }
__device__ __forceinline__ df acc_df(const Acc &s) { return dev::fast_two_sum(s.hi, s.lo); }
__device__ __forceinline__ df scale2(df a, float s) { return {a.hi * s, a.lo * s}; }   // s a power of two, or +-1

// Sum over the warp of 32 values per lane: lane l returns the sum of value l
// (31 additions instead of 5 per value).
__device__ __forceinline__ Acc warp_transpose_sum(Acc (&v)[32], int lane) {
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const bool up = lane & s;
#pragma unroll
        for (int i = 0; i < s; ++i) {
            const Acc keep = up ? v[i + s] : v[i], send = up ? v[i] : v[i + s];
            const float h = __shfl_xor_sync(0xffffffffu, send.hi, s), l = __shfl_xor_sync(0xffffffffu, send.lo, s);
            const df t = dev::two_sum(keep.hi, h);
            v[i] = Acc{t.hi, __fadd_rn(__fadd_rn(keep.lo, l), t.lo)};
        }
    }
    return v[0];
}

constexpr int kAT = 256;   // threads of the double-float reverse pass
__global__ void __launch_bounds__(kAT, 512 / kAT)
adjoint_df64_kernel(int64_t N, int64_t M, const double *__restrict__ src, const double *__restrict__ fpts,
                    const double2 *__restrict__ w, const double2 *__restrict__ p, const float *__restrict__ rec,
                    int stride, int nidx_off, const __grid_constant__ dev::RuleInfo ri,
                    const double *__restrict__ coords, const double2 *__restrict__ Y, int64_t E, int S,
                    const float *__restrict__ tab, int qmax, const __grid_constant__ AdjView v64, double kre,
                    double rhock, df64::DfDegrees deg, int chunk, double *__restrict__ sums,
                    double *__restrict__ dX) {
    extern __shared__ __align__(16) float smemf[];
    float *s_tab = smemf;                                        // 3 qmax kAdjTab
    float *s_rec = s_tab + 3 * qmax * kAdjTab;                   // chunk * stride
    float4 *s_ph = reinterpret_cast<float4 *>(s_rec + (size_t)chunk * stride);   // chunk * 3 qmax: p(x_q)
    float *s_el = reinterpret_cast<float *>(s_ph + (size_t)chunk * 3 * qmax);    // chunk * 32: e_b, G0, centroid
    __shared__ dev::RuleInfo s_ri;
    if (threadIdx.x == 0) s_ri = ri;
    for (int t = threadIdx.x; t < 3 * qmax * kAdjTab; t += kAT) s_tab[t] = tab[t];
    const int lane = threadIdx.x & 31;
    const int s = blockIdx.y;
    const int64_t e0 = (int64_t)s * E / S, e1 = (int64_t)(s + 1) * E / S;
    const df K = dd::to_df(kre), K2 = dd::to_df(kre * kre);
    const float kf = K.hi, k3 = third(kre, K), k23 = third(kre * kre, K2);

    const int64_t row = (int64_t)blockIdx.x * kAT + threadIdx.x;
    const bool active = row < N + M, node = row < N;   // collocation row, else field row
    const float aF = node ? 1.0f : -1.0f;              // alpha_F, and the sign of alpha_G's factor
    double tx = 0, ty = 0, tz = 0;
    double2 wv = make_double2(0, 0), pv = wv;
    if (active) {
        const double *t = node ? src + 3 * row : fpts + 3 * (row - N);
        tx = t[0];
        ty = t[1];
        tz = t[2];
        wv = w[row];
        if (node) pv = p[row];
    }
    const df cwr = dd::to_df(wv.x), cwi = dd::to_df(-wv.y);
    const df sc = dd::to_df(node ? wv.x * pv.x + wv.y * pv.y : 0.0);   // Re conj(w) p_i
    Acc gt[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    for (int64_t cb = e0; cb < e1; cb += chunk) {
        const int n = (int)min((int64_t)chunk, e1 - cb);
        __syncthreads();
        {
            const float4 *a = reinterpret_cast<const float4 *>(rec + cb * stride);
            float4 *b = reinterpret_cast<float4 *>(s_rec);
            for (int t = threadIdx.x; t < n * stride / 4; t += kAT) b[t] = a[t];
        }
        __syncthreads();
        for (int t = threadIdx.x; t < n * 3 * qmax; t += kAT) {   // p at the points, in FP64
            const int el = t / (3 * qmax), c = (t - el * 3 * qmax) / qmax, q = t - el * 3 * qmax - c * qmax;
            const int32_t *nid = reinterpret_cast<const int32_t *>(s_rec + (size_t)el * stride + nidx_off);
            if (q >= s_ri.Q[c]) continue;
            double re = 0, im = 0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const double Na = v64.phi[((size_t)c * v64.qmax + q) * 3 + a];
                const double2 pa = p[nid[a]];
                re += Na * pa.x;
                im += Na * pa.y;
            }
            const df x = dd::to_df(re), y = dd::to_df(im);
            s_ph[t] = make_float4(x.hi, x.lo, y.hi, y.lo);
        }
        for (int t = threadIdx.x; t < n * 11; t += kAT) {         // X_b - centroid, rhock (Im Y, -Re Y)
            const int el = t / 11, j = t - el * 11;
            const float *r = s_rec + (size_t)el * stride;
            double x;
            if (j < 9) {
                const int b = j / 3, k = j - 3 * b;
                const double cen = (double)r[k] + (double)r[3 + k];
                x = coords[3 * (int64_t)reinterpret_cast<const int32_t *>(r + nidx_off)[b] + k] - cen;
            } else {
                const double2 y = Y[cb + el];
                x = j == 9 ? rhock * y.y : -rhock * y.x;
            }
            const df h = dd::to_df(x);
            s_el[32 * el + 2 * j] = h.hi;
            s_el[32 * el + 2 * j + 1] = h.lo;
            if (j < 3)
                reinterpret_cast<double *>(s_el + 32 * el + 24)[j] = (double)r[j] + (double)r[3 + j];   // centroid
        }
        __syncthreads();

#pragma unroll 1
        for (int el = 0; el < n; ++el) {
            // (the warps stay together: the loop is longer than the instruction caches,
            // and each would fetch it for itself)
            __syncthreads();
            const float *r = s_rec + (size_t)el * stride;
            const float2 *se = reinterpret_cast<const float2 *>(s_el + 32 * el);
            const df G0r{se[9].x, se[9].y}, G0i{se[10].x, se[10].y};
            Acc v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = Acc{0.f, 0.f};
            if (active) {
                // D = centroid - t in FP64 before it is split: of absolute coordinates
                // rounded to float pairs it would lose 2^-48 |x|
                const double *cen = reinterpret_cast<const double *>(s_el + 32 * el + 24);
                const double ax = cen[0] - tx, ay = cen[1] - ty, az = cen[2] - tz;
                const mixed::PairSetup P = mixed::pair_setup<3>(r, r[6], dd::to_df(ax), dd::to_df(ay), dd::to_df(az));
                df r0, ri0;
                dd::sqrt_rcp_df(dev::df_add(dev::df_add(dev::df_sqr(P.Dxd), dev::df_sqr(P.Dyd)), dev::df_sqr(P.Dzd)),
                                r0, ri0);
                Acc m[6], sb[3], sg{0.f, 0.f}, szr{0.f, 0.f}, szi{0.f, 0.f};
#pragma unroll
                for (int a = 0; a < 6; ++a) m[a] = Acc{0.f, 0.f};
#pragma unroll
                for (int a = 0; a < 3; ++a) sb[a] = Acc{0.f, 0.f};
                if (P.deferred || !(fabsf(kf * r0.hi) < df64::kDfMaxPhase)) {
                    const cd g0 = {(double)G0r.hi + (double)G0r.lo, (double)G0i.hi + (double)G0i.lo};
                    const AdjPair o = adjoint_pair_fp64(
                        v64, cb + el, tx, ty, tz,
                        cd{(double)cwr.hi + (double)cwr.lo, (double)cwi.hi + (double)cwi.lo},
                        (double)sc.hi + (double)sc.lo, (double)aF, (double)aF, g0, p, kre);
                    auto acc_of = [](double x) {
                        const df t = dd::to_df(x);
                        return Acc{t.hi, t.lo};
                    };
#pragma unroll
                    for (int a = 0; a < 6; ++a) m[a] = acc_of(o.M[a]);
#pragma unroll
                    for (int a = 0; a < 3; ++a) sb[a] = acc_of(o.SB[a]);
                    sg = acc_of(o.SG);
                    szr = acc_of(o.SZr);
                    szi = acc_of(o.SZi);
                } else {
                    // e^{i k r0}: phase and quadrant in FP64 (fifteen operations of an
                    // otherwise idle pipe), series in double-float
                    df E0r, E0i;
                    {
                        const double q2 = ax * ax + ay * ay + az * az;
                        const double x = kre * (q2 * rsqrt(q2));
                        const double nq = rint(x * 0.63661977236758134308);   // 2 / pi
                        const double y = fma(-nq, 6.123233995736766036e-17, fma(-nq, 1.57079632679489655800, x));
                        dd::sincos_df(dd::to_df(y), E0i, E0r);
                        const int quad = ((int)nq) & 3;
                        if (quad & 1) {
                            const df t = E0r;
                            E0r = dd::neg(E0i);
                            E0i = t;
                        }
                        if (quad & 2) {
                            E0r = dd::neg(E0r);
                            E0i = dd::neg(E0i);
                        }
                    }
                    // conj(w) e^{i k r0}
                    const df hr = dev::df_sub(dev::df_mul(cwr, E0r), dev::df_mul(cwi, E0i));
                    const df hi = dev::df_add(dev::df_mul(cwr, E0i), dev::df_mul(cwi, E0r));
                    const int c = P.c, Q = s_ri.Q[c];
                    const float4 *g4 = reinterpret_cast<const float4 *>(r + s_ri.off[c]);
                    const float4 *ph = s_ph + ((size_t)el * 3 + c) * qmax;
                    const float4 *tb = reinterpret_cast<const float4 *>(s_tab + (size_t)c * qmax * kAdjTab);
#pragma unroll 1
                    for (int q = 0; q < Q; ++q) {
                        const float4 A = g4[4 * q], B4 = g4[4 * q + 1], Cn = g4[4 * q + 2], Dn = g4[4 * q + 3];
                        const df ox{A.x, B4.x}, oy{A.y, B4.y}, oz{A.z, B4.z};
                        const df dx = dev::df_add(P.Dxd, ox), dy = dev::df_add(P.Dyd, oy), dz = dev::df_add(P.Dzd, oz);
                        df rr, ri1;
                        dd::sqrt_rcp_df(dev::df_add(dev::df_add(dev::df_sqr(dx), dev::df_sqr(dy)), dev::df_sqr(dz)),
                                        rr, ri1);
                        // r - r0 = (2 D.o + |o|^2) / (r + r0), free of cancellation: at a
                        // distance of 10 the difference of two rounded lengths would cost
                        // the phase 1e-13
                        const df Do = dev::df_add(dev::df_add(dev::df_mul(P.Dxd, ox), dev::df_mul(P.Dyd, oy)),
                                                  dev::df_mul(P.Dzd, oz));
                        const df dr = dev::df_mul(dev::df_add(scale2(Do, 2.0f), df{Cn.w, Dn.w}),
                                                  dd::rcp(dev::df_add(rr, r0)));
                        df ct, st;
                        df64::rotation_df64(mul_k(K, k3, dr), deg, ct, st);
                        const float4 pq = ph[q];
                        const df pr{pq.x, pq.y}, pi{pq.z, pq.w};
                        // z = conj(w) e^{i k r0} (p(x_q) e^{i k (r - r0)})
                        const df ar = dev::df_sub(dev::df_mul(pr, ct), dev::df_mul(pi, st));
                        const df ai = dev::df_add(dev::df_mul(pr, st), dev::df_mul(pi, ct));
                        const df zr = dev::df_sub(dev::df_mul(hr, ar), dev::df_mul(hi, ai));
                        const df zi = dev::df_add(dev::df_mul(hr, ai), dev::df_mul(hi, ar));
                        const df kr = mul_k(K, k3, rr);
                        const df ri2 = dev::df_sqr(ri1);
                        const df t3 = dev::df_sub(scale2(dev::df_add(zr, dev::df_mul(kr, zi)), aF), sc);
                        const df gr = dev::df_sub(dev::df_mul(zr, G0r), dev::df_mul(zi, G0i));
                        const df gi = dev::df_add(dev::df_mul(zr, G0i), dev::df_mul(zi, G0r));
                        const df gp = scale2(dev::df_add(gr, dev::df_mul(kr, gi)), -aF);
                        const df wr = dev::df_mul(df{A.w, B4.w}, ri1);
                        const df dh = dev::df_mul(
                            dev::df_add(dev::df_add(dev::df_mul(dx, df{Cn.x, Dn.x}), dev::df_mul(dy, df{Cn.y, Dn.y})),
                                        dev::df_mul(dz, df{Cn.z, Dn.z})), ri1);   // -(d.n)/r
                        const df tr = dev::df_mul(t3, ri2);
                        // aF k^2 z_r - 3 t3 / r^2 (3 x = 2 x + x)
                        const df q1 = dev::df_sub(scale2(mul_k(K2, k23, zr), aF), dev::df_add(scale2(tr, 2.0f), tr));
                        const df A1 = dev::df_mul(dev::df_mul(wr, ri1),
                                                  dev::df_sub(dev::df_mul(gp, ri1), dev::df_mul(dh, q1)));
                        const df B1 = dev::df_mul(wr, tr);
                        const float4 t0 = tb[5 * q], t1 = tb[5 * q + 1], t2 = tb[5 * q + 2], t4 = tb[5 * q + 3],
                                     t5 = tb[5 * q + 4];
                        acc_prod(m[0], A1, df{t0.x, t0.y});
                        acc_prod(m[1], A1, df{t0.z, t0.w});
                        acc_prod(m[2], A1, df{t1.x, t1.y});
                        acc_prod(m[3], A1, df{t1.z, t1.w});
                        acc_prod(m[4], A1, df{t2.x, t2.y});
                        acc_prod(m[5], A1, df{t2.z, t2.w});
                        acc_prod(sb[0], B1, df{t4.x, t4.y});
                        acc_prod(sb[1], B1, df{t4.z, t4.w});
                        acc_prod(sb[2], B1, df{t5.x, t5.y});
                        const df ws = scale2(wr, aF);
                        acc_prod(sg, ws, gr);
                        acc_prod(szr, ws, zr);
                        acc_prod(szi, ws, zi);
                    }
                }
                // over the element: M, D M_a, SB, D SB, SG, SZ; and the row's gradient
                // -(sum_q A' d + B n)
                df mm[6], mb[3], sbd[3];
#pragma unroll
                for (int a = 0; a < 6; ++a) mm[a] = acc_df(m[a]);
                mb[0] = dev::df_add(dev::df_add(mm[0], mm[3]), mm[4]);
                mb[1] = dev::df_add(dev::df_add(mm[1], mm[3]), mm[5]);
                mb[2] = dev::df_add(dev::df_add(mm[2], mm[4]), mm[5]);
#pragma unroll
                for (int a = 0; a < 3; ++a) sbd[a] = acc_df(sb[a]);
                const df sbt = dev::df_add(dev::df_add(sbd[0], sbd[1]), sbd[2]);
                const df mt = dev::df_add(dev::df_add(mb[0], mb[1]), mb[2]);
                const df D[3] = {P.Dxd, P.Dyd, P.Dzd};
#pragma unroll
                for (int a = 0; a < 6; ++a) dd::acc_add(v[a], mm[a]);
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int k = 0; k < 3; ++k) acc_prod(v[6 + 3 * a + k], D[k], mb[a]);
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    dd::acc_add(v[15 + a], sbd[a]);
                    acc_prod(v[18 + a], D[a], sbt);
                }
                dd::acc_add(v[21], acc_df(sg));
                dd::acc_add(v[22], acc_df(szr));
                dd::acc_add(v[23], acc_df(szi));
                if (node) {
                    const float4 Cn = *reinterpret_cast<const float4 *>(r + s_ri.off[0] + 8);
                    const float4 Dn = *reinterpret_cast<const float4 *>(r + s_ri.off[0] + 12);
                    const df nr[3] = {{Cn.x, Dn.x}, {Cn.y, Dn.y}, {Cn.z, Dn.z}};   // -n
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        acc_prod(gt[k], dd::neg(D[k]), mt);
                        acc_prod(gt[k], nr[k], sbt);
#pragma unroll
                        for (int b = 0; b < 3; ++b) {
                            const float2 eb = se[3 * b + k];
                            acc_prod(gt[k], df{-eb.x, -eb.y}, mb[b]);
                        }
                    }
                }
            }
            const Acc t = warp_transpose_sum(v, lane);
            if (lane < kAdjSums) atomicAdd(sums + (size_t)(cb + el) * kAdjSums + lane, dd::acc_value(t));
        }
    }
    if (node)
#pragma unroll
        for (int k = 0; k < 3; ++k) atomicAdd(&dX[3 * row + k], dd::acc_value(gt[k]));
}

// Vertex gradients and admittance sensitivities of every element from its sums.
__global__ void adjoint_finish_kernel(const double *__restrict__ sums, const double *__restrict__ coords,
                                      const int32_t *__restrict__ topo, const int32_t *__restrict__ order, int64_t E,
                                      double rhock, double *__restrict__ dX, double2 *__restrict__ sY) {
    const int64_t pe = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pe >= E) return;
    const int64_t e = order[pe];
    const double *s = sums + pe * kAdjSums;
    double X[3][3], cen[3], n[3], eb[3][3], u[3], v[3];
    for (int b = 0; b < 3; ++b)
        for (int k = 0; k < 3; ++k) X[b][k] = coords[3 * (int64_t)topo[3 * e + b] + k];
    for (int k = 0; k < 3; ++k) {
        cen[k] = X[0][k] / 3.0;
        cen[k] += X[1][k] / 3.0;
        cen[k] += X[2][k] / 3.0;
        const float hi = (float)cen[k];   // as the records hold it
        cen[k] = (double)hi + (double)(float)(cen[k] - (double)hi);
        u[k] = X[1][k] - X[0][k];
        v[k] = X[2][k] - X[0][k];
        for (int b = 0; b < 3; ++b) eb[b][k] = X[b][k] - cen[k];
    }
    n[0] = u[1] * v[2] - u[2] * v[1];
    n[1] = u[2] * v[0] - u[0] * v[2];
    n[2] = u[0] * v[1] - u[1] * v[0];
    const double J = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    for (int k = 0; k < 3; ++k) n[k] /= J;
    const int ix[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
    double g[3][3], Gn[3];
    for (int k = 0; k < 3; ++k) {
        Gn[k] = s[18 + k] + n[k] * s[21];
        for (int a = 0; a < 3; ++a) {
            double t = s[6 + 3 * a + k] + n[k] * s[15 + a];
            for (int b = 0; b < 3; ++b) t += eb[b][k] * s[ix[a][b]];
            g[a][k] = t;
            Gn[k] += eb[a][k] * s[15 + a];
        }
    }
    for (int k = 0; k < 3; ++k) Gn[k] /= J;
    // nn = u x v: dL/du = v x Gn, dL/dv = Gn x u
    const double au[3] = {v[1] * Gn[2] - v[2] * Gn[1], v[2] * Gn[0] - v[0] * Gn[2], v[0] * Gn[1] - v[1] * Gn[0]};
    const double av[3] = {Gn[1] * u[2] - Gn[2] * u[1], Gn[2] * u[0] - Gn[0] * u[2], Gn[0] * u[1] - Gn[1] * u[0]};
    for (int k = 0; k < 3; ++k) {
        atomicAdd(&dX[3 * (int64_t)topo[3 * e] + k], g[0][k] - au[k] - av[k]);
        atomicAdd(&dX[3 * (int64_t)topo[3 * e + 1] + k], g[1][k] + au[k]);
        atomicAdd(&dX[3 * (int64_t)topo[3 * e + 2] + k], g[2][k] + av[k]);
    }
    // sum of sgn z W / r times -i rhock
    sY[e] = make_double2(rhock * s[23], -rhock * s[22]);
}

inline unsigned nblocks(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// Whether the double-float kernel's values stay clear of the ends of FP32's range.
// They go with the adjoint pressure over the mesh size L (a gradient's terms, and
// about 2^-14 of it per point); the error term of a product of pairs is 2^-72 of
// it.  Largest adjoint pressure over L and error against the FP64 kernel: 2^-37
// 3e-14, 2^-47 5e-14, 2^-53 3e-10, 2^-57 6e-11 .. 1e-4.
bool double_float_range(const Ctx &c, const std::vector<std::complex<double>> &lam,
                        const std::vector<std::complex<double>> &pf, const AdjointArgs &a) {
    auto largest = [](const std::vector<std::complex<double>> &v) {
        double m = 0.0;
        for (const auto &x : v) m = std::max(m, std::max(std::fabs(x.real()), std::fabs(x.imag())));
        return m;
    };
    const double l = largest(lam), p = largest(pf);
    double z = INFINITY;
    for (int64_t e = 0; e < 2 * c.n_elements; e += 2)
        z = std::min(z, std::max(std::fabs(a.Z[e]), std::fabs(a.Z[e + 1])));
    return l >= std::ldexp(1.0, c.fx_exp - 40) && l <= 0x1p40 && p <= 0x1p40 &&
           std::fabs(a.rho_c * a.k_re) <= 0x1p60 * z;
}

}  // namespace

void run_adjoint(Ctx &c, const AdjointArgs &a, AdjointOut &out) {
    if (c.shape_kind != BIE_TRI_LINEAR || c.physics_kind != BIE_TRI_LINEAR)
        fail(BIE_ERR_UNSUPPORTED, "the adjoint supports 3-node triangles with vertex physics");
    if (c.n_sources != c.n_coords || c.sources != c.coords || c.ptopo != c.topo)
        fail(BIE_ERR_UNSUPPORTED, "the adjoint needs collocation nodes identical to the vertices");
    const int64_t N = c.n_sources, E = c.n_elements, M = a.n_field;
    if (a.k_im != 0.0) fail(BIE_ERR_UNSUPPORTED, "the adjoint supports real wavenumbers");
    // device buffers (allocated per call; the adjoint runs once per design step)
    struct Buf {
        void *p = nullptr;
        explicit Buf(size_t b) { BIE_CUDA(cudaMalloc(&p, std::max<size_t>(b, 16))); }
        ~Buf() { cudaFree(p); }
        double2 *d2() const { return static_cast<double2 *>(p); }
        double *d() const { return static_cast<double *>(p); }
        int32_t *i32() const { return static_cast<int32_t *>(p); }
    };
    Buf A((size_t)N * N * 16), G((size_t)N * N * 16), B((size_t)M * N * 16), Gx((size_t)M * N * 16);
    Buf Cv(N * 16), Y(E * 16), Zd(E * 16), ord(E * 4), fp(M * 24), pI(N * 16), pIf(M * 16);
    Buf p(N * 16), pf(M * 16), rhs(N * 16), lam(N * 16), w((N + M) * 16), dX(3 * N * 8), sY(E * 16);
    Buf tab(4 * 3 * 64 * 8);
    cudaStream_t st = c.stream;
    BIE_CUDA(cudaMemcpyAsync(Zd.p, a.Z, E * 16, cudaMemcpyHostToDevice, st));
    BIE_CUDA(cudaMemcpyAsync(ord.p, c.order.data(), E * 4, cudaMemcpyHostToDevice, st));
    BIE_CUDA(cudaMemcpyAsync(fp.p, a.field, M * 24, cudaMemcpyHostToDevice, st));
    admittance_kernel<<<nblocks(E), 256, 0, st>>>(Zd.d2(), ord.i32(), E, Y.d2());
    BIE_CUDA(cudaGetLastError());
    if (!c.d_coords) {
        BIE_CUDA(cudaMalloc(&c.d_coords, c.coords.size() * sizeof(double)));
        BIE_CUDA(cudaMemcpy(c.d_coords, c.coords.data(), c.coords.size() * sizeof(double), cudaMemcpyHostToDevice));
        BIE_CUDA(cudaMalloc(&c.d_topo, c.topo.size() * sizeof(int32_t)));
        BIE_CUDA(cudaMemcpy(c.d_topo, c.topo.data(), c.topo.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    }
    // double-float holds squares and cubes of lengths: mesh sizes within 2^+-30
    // (gradient error 4e-14 at 2^-43, 3e-12 to 8e-12 at 2^-50)
    const bool use_df = a.precision == BIE_PREC_DF64 && c.fx_ok && std::abs(c.fx_exp) <= 30;
    // -i rho c k and +i rho c k (k real)
    const double2 aAc = make_double2(0.0, -a.rho_c * a.k_re);
    const double2 aBc = make_double2(0.0, a.rho_c * a.k_re);
    // ---- forward: A, B ----------------------------------------------------------
    {
        // |Y| < 2^400 for the fixed-point assembly (an infinite Y, from |Z|^2 = 0, is not)
        bool bounded = true;
        for (int64_t e = 0; e < 2 * E; e += 2)
            bounded = bounded && std::max(std::fabs(a.Z[e]), std::fabs(a.Z[e + 1])) > 0x1p-399;
        AssembleArgs s{a.k_re, a.k_im, c.d_sources, N, BIE_F | BIE_G | BIE_C, A.d(), G.d(), Cv.d()};
        s.g_weight = Y.d();
        s.g_weight_bounded = bounded;
        if (!(use_df && launch_assemble_df64(c, s))) launch_assemble_fp64(c, s);
        combine_system_kernel<<<std::min<unsigned>(nblocks(N * N), 65535u), 256, 0, st>>>(
            A.d2(), G.d2(), aAc, Cv.d2(), N, N);
        BIE_CUDA(cudaGetLastError());
        AssembleArgs f{a.k_re, a.k_im, fp.d(), M, BIE_F | BIE_G, B.d(), Gx.d(), nullptr};
        f.g_weight = Y.d();
        f.g_weight_bounded = bounded;
        if (!(use_df && launch_assemble_df64(c, f))) launch_assemble_fp64(c, f);
        // stored: F_x - i rho c k G_x  (= -B)
        combine_system_kernel<<<std::min<unsigned>(nblocks(M * N), 65535u), 256, 0, st>>>(
            B.d2(), Gx.d2(), make_double2(-aBc.x, -aBc.y), nullptr, M, N);
        BIE_CUDA(cudaGetLastError());
    }
    incident_kernel<<<nblocks(N), 256, 0, st>>>(c.d_sources, N, a.k_re, a.k_im, a.dir[0], a.dir[1],
                                                 a.dir[2], pI.d2());
    incident_kernel<<<nblocks(M), 256, 0, st>>>(fp.d(), M, a.k_re, a.k_im, a.dir[0], a.dir[1], a.dir[2],
                                                 pIf.d2());
    BIE_CUDA(cudaGetLastError());
    bie_gmres_opts go{};
    go.reltol = a.reltol > 0 ? a.reltol : 1e-13;
    go.restart = 60;
    go.maxiter = (int)std::min<int64_t>(N, 5000);
    go.precision = BIE_PREC_FP64;
    bie_gmres_info gi{};
    bie_operator op{};
    op.kind = BIE_OP_DENSE;
    op.A = A.d();
    op.scale_re = 1.0;
    run_gmres(c, op, pI.d(), p.d(), go, gi);
    out.forward_iterations = gi.iterations;
    out.forward_converged = gi.converged;
    // The B buffer holds F_x - i rho c k G_x = -B, so p_f = p_I(x_f) - (stored) p.
    {
        Buf tmp(M * 16), zero(M * 16);
        BIE_CUDA(cudaMemsetAsync(zero.p, 0, M * 16, st));
        small_gemv_kernel<<<nblocks(M * 32), 256, 0, st>>>(B.d2(), M, N, p.d2(), zero.d2(), tmp.d2());
        BIE_CUDA(cudaGetLastError());
        std::vector<std::complex<double>> ht(M), hi(M);
        BIE_CUDA(cudaMemcpyAsync(ht.data(), tmp.p, M * 16, cudaMemcpyDeviceToHost, st));
        BIE_CUDA(cudaMemcpyAsync(hi.data(), pIf.p, M * 16, cudaMemcpyDeviceToHost, st));
        BIE_CUDA(cudaStreamSynchronize(st));
        double J = 0;
        std::vector<std::complex<double>> hpf(M);
        for (int64_t j = 0; j < M; ++j) {
            hpf[j] = hi[j] - ht[j];
            J += std::norm(hpf[j]);
        }
        out.J = J;
        if (a.pf) std::copy(hpf.begin(), hpf.end(), reinterpret_cast<std::complex<double> *>(a.pf));
        BIE_CUDA(cudaMemcpyAsync(pf.p, hpf.data(), M * 16, cudaMemcpyHostToDevice, st));
        BIE_CUDA(cudaStreamSynchronize(st));
    }
    if (!a.dX && !a.dZ) return;
    // ---- adjoint: A^H lambda = B^H p_f  (B^H p_f = -(stored)^H p_f) ---------------
    adjoint_rhs_kernel<<<nblocks(N), 256, 0, st>>>(B.d2(), M, N, pf.d2(), rhs.d2());
    BIE_CUDA(cudaGetLastError());
    {
        std::vector<std::complex<double>> hr(N);
        BIE_CUDA(cudaMemcpyAsync(hr.data(), rhs.p, N * 16, cudaMemcpyDeviceToHost, st));
        BIE_CUDA(cudaStreamSynchronize(st));
        for (auto &v : hr) v = -v;
        BIE_CUDA(cudaMemcpyAsync(rhs.p, hr.data(), N * 16, cudaMemcpyHostToDevice, st));
        BIE_CUDA(cudaStreamSynchronize(st));
    }
    conj_transpose_kernel<<<dim3((unsigned)((N + 31) / 32), (unsigned)((N + 31) / 32)), dim3(32, 8), 0, st>>>(
        A.d2(), G.d2(), N);   // G buffer reused for A^H
    BIE_CUDA(cudaGetLastError());
    op.A = G.d();
    run_gmres(c, op, rhs.d(), lam.d(), go, gi);
    out.adjoint_iterations = gi.iterations;
    out.adjoint_converged = gi.converged;
    // ---- reverse pass ----------------------------------------------------------------
    {
        std::vector<std::complex<double>> hl(N), hw(N + M), hp(M);
        BIE_CUDA(cudaMemcpyAsync(hl.data(), lam.p, N * 16, cudaMemcpyDeviceToHost, st));
        BIE_CUDA(cudaMemcpyAsync(hp.data(), pf.p, M * 16, cudaMemcpyDeviceToHost, st));
        BIE_CUDA(cudaStreamSynchronize(st));
        for (int64_t i = 0; i < N; ++i) hw[i] = -hl[i];
        for (int64_t j = 0; j < M; ++j) hw[N + j] = hp[j];
        BIE_CUDA(cudaMemcpyAsync(w.p, hw.data(), (N + M) * 16, cudaMemcpyHostToDevice, st));
        // rule table: 3 corner rules, 4 doubles per point (N1 N2 N3 w)
        std::vector<double> ht;
        RuleTab rt{};
        for (int r = 0; r < 3; ++r) {
            rt.off[r] = (int)(ht.size() / 4);
            rt.Q[r] = c.rules[r].size();
            for (int q = 0; q < rt.Q[r]; ++q) {
                double Nv[3];
                shape_values(BIE_TRI_LINEAR, c.rules[r].u[q], c.rules[r].v[q], Nv);
                ht.push_back(Nv[0]);
                ht.push_back(Nv[1]);
                ht.push_back(Nv[2]);
                ht.push_back(c.rules[r].w[q]);
            }
        }
        BIE_CUDA(cudaMemcpyAsync(tab.p, ht.data(), ht.size() * 8, cudaMemcpyHostToDevice, st));
        BIE_CUDA(cudaMemsetAsync(dX.p, 0, 3 * N * 8, st));
        BIE_CUDA(cudaMemsetAsync(sY.p, 0, E * 16, st));
        const double rhock_re = a.rho_c * a.k_re;
        df64::DfDegrees deg{};
        // (a caller of BIE_PREC_FP64 gets FP64 here too)
        if (use_df && double_float_range(c, hl, hp, a) &&
            df64::df_degrees(std::fabs(a.k_re) * c.df_rho_max, 0.0, deg)) {
            deg.tab = reinterpret_cast<const float4 *>(c.d_phase_tab);
            const RecordLayout &L = c.lay;
            const Df64Layout &X = c.dlay;
            AdjView v{c.d_records, L.stride, L.nidx_off, L.qmax, c.d_phi, c.d_xtrig, {}};
            dev::RuleInfo ri{};
            for (int r = 0; r < 3; ++r) {
                ri.Q[r] = v.ri.Q[r] = L.Q[r];
                ri.off[r] = X.rule_off[r];
                v.ri.off[r] = L.rule_off[r];
            }
            // N_a N_b and N_a per rule point as hi, lo
            std::vector<float> tb((size_t)3 * L.qmax * kAdjTab, 0.f);
            for (int r = 0; r < 3; ++r)
                for (int q = 0; q < L.Q[r]; ++q) {
                    const double *Nv = &c.phi[((size_t)r * L.qmax + q) * 3];
                    const double x[10] = {Nv[0] * Nv[0], Nv[1] * Nv[1], Nv[2] * Nv[2], Nv[0] * Nv[1],
                                          Nv[0] * Nv[2], Nv[1] * Nv[2], Nv[0], Nv[1], Nv[2], 0.0};
                    float *t = &tb[((size_t)r * L.qmax + q) * kAdjTab];
                    for (int j = 0; j < 10; ++j) {
                        t[2 * j] = (float)x[j];
                        t[2 * j + 1] = (float)(x[j] - (double)t[2 * j]);
                    }
                }
            Buf dtab(tb.size() * 4), sums((size_t)E * kAdjSums * 8);
            BIE_CUDA(cudaMemcpyAsync(dtab.p, tb.data(), tb.size() * 4, cudaMemcpyHostToDevice, st));
            BIE_CUDA(cudaMemsetAsync(sums.p, 0, (size_t)E * kAdjSums * 8, st));
            // chunks of ~48 KB: two blocks per SM with room for L1
            const size_t el_bytes = (size_t)X.stride * 4 + (size_t)3 * L.qmax * 16 + 32 * 4;
            const int chunk = (int)std::max<size_t>(1, std::min<size_t>(32, (48u << 10) / el_bytes));
            const size_t smem = tb.size() * 4 + chunk * el_bytes;
            const int64_t tiles = (N + M + kAT - 1) / kAT;
            int S = 1;
            // many small blocks: their cost differs with the near pairs in them (blocks
            // of 128 threads: 13.5 ms at 64 blocks per SM, 14.0 at 32, 14.9 at 16, 16.4 at 8)
            while (tiles * S < 64LL * c.num_sms && S * 2 * 8 <= E) S *= 2;
            BIE_CUDA(cudaFuncSetAttribute(adjoint_df64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            adjoint_df64_kernel<<<dim3((unsigned)tiles, (unsigned)S), kAT, smem, st>>>(
                N, M, c.d_sources, fp.d(), w.d2(), p.d2(), c.d_drecords, X.stride, X.nidx_off, ri, c.d_coords, Y.d2(),
                E, S, static_cast<const float *>(dtab.p), L.qmax, v, a.k_re, rhock_re, deg, chunk, sums.d(), dX.d());
            BIE_CUDA(cudaGetLastError());
            adjoint_finish_kernel<<<nblocks(E), 256, 0, st>>>(sums.d(), c.d_coords, c.d_topo, ord.i32(), E, rhock_re,
                                                              dX.d(), sY.d2());
            BIE_CUDA(cudaGetLastError());
            BIE_CUDA(cudaStreamSynchronize(st));   // the call's buffers go out of scope
        } else {   // FP64, or values or phase rotations beyond the double-float kernel's
            int S = 1;
            const int64_t tiles = (N + M + kT - 1) / kT;
            while (tiles * S < 8LL * c.num_sms && S < 256 && S * 2 <= E) S *= 2;
            dim3 grid((unsigned)tiles, (unsigned)S);
            adjoint_grad_kernel<false><<<grid, kT, 0, st>>>(N, M, c.d_sources, fp.d(), w.d2(), p.d2(),
                                                            c.d_coords, c.d_topo, ord.i32(), Y.d2(), E, S,
                                                            tab.d(), rt, c.d_xtrig, a.k_re, a.k_im, rhock_re,
                                                            dX.d(), sY.d2());
            BIE_CUDA(cudaGetLastError());
        }
        std::vector<double> hdX(3 * N);
        std::vector<std::complex<double>> hs(E), hpI(N);
        BIE_CUDA(cudaMemcpyAsync(hdX.data(), dX.p, 3 * N * 8, cudaMemcpyDeviceToHost, st));
        BIE_CUDA(cudaMemcpyAsync(hs.data(), sY.p, E * 16, cudaMemcpyDeviceToHost, st));
        BIE_CUDA(cudaMemcpyAsync(hpI.data(), pI.p, N * 16, cudaMemcpyDeviceToHost, st));
        BIE_CUDA(cudaStreamSynchronize(st));
        if (a.dX) {
            const std::complex<double> ik(-a.k_im, a.k_re);
            for (int64_t i = 0; i < N; ++i) {
                // 2 Re[conj(lambda_i) d p_I / d x_i],  d p_I / d x = -i k d p_I
                const std::complex<double> s = std::conj(hl[i]) * (-ik) * hpI[i];
                for (int k = 0; k < 3; ++k) a.dX[3 * i + k] = 2.0 * hdX[3 * i + k] + 2.0 * s.real() * a.dir[k];
            }
        }
        if (a.dZ) {
            const std::complex<double> *Z = reinterpret_cast<const std::complex<double> *>(a.Z);
            std::complex<double> *dZ = reinterpret_cast<std::complex<double> *>(a.dZ);
            for (int64_t e = 0; e < E; ++e) dZ[e] = -2.0 * std::conj(hs[e] / (Z[e] * Z[e]));
        }
    }
}

}  // namespace bie
