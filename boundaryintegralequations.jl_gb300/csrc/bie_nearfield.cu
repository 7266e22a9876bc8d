// Near-field (sparse) FP64 assembly: the GPU counterpart of
// sparse_assemble_parallel! (src/3d/assembly_collocation_losses.jl:200-405, with
// sparse_computing_integrals! :158-186) and of the coarse partial assembly
// partial_assemble_parallel! (src/3d/fast_multipole_method.jl:11-81).
//
// One warp per (collocation node, connected element) pair: the warp picks the
// rule of the geometry node nearest to the target (find_closest_corner on the
// element's geometry nodes, Julia hypot semantics) — or the coarse Gauss rule —
// and its lanes stride over the rule's points (3711 points for a corner rule,
// 10623 for an edge-midpoint rule at offset 0).  Per point the geometry is
// interpolated from the element's nodes (tabulated shape functions and
// derivatives), the jacobian and negated unit normal formed as in jacobian!
// (src/3d/jacobian.jl:78-87), and the F and G integrands of kernels.jl:13-37
// accumulated per physics node.  A warp-shuffle reduction gives the element's
// contributions, which the lanes add (FP64 atomics) to the pair's CSR slots.
// FP64 throughout (roots, divisions, sine, cosine and exponential at FP64 accuracy
// on the integer pipes): these are the singular and near-singular integrals.
#include "bie_internal.h"
#include "bie_device.cuh"
#include "bie_fixmath.cuh"

namespace bie {

namespace {

constexpr double kInv4Pi = 0.07957747154594767;

struct RuleSet {
    int64_t off[kMaxRules];
    int q[kMaxRules];
    int64_t coarse_off;
    int coarse_q;
};

// Sums of V = 16 or 32 values over the warp's lanes, halving the values with
// each exchange (V adds instead of 5 V): lane l gets value l (32) or l / 2 (16).
template <int V>
__device__ __forceinline__ double warp_sums(double (&v)[V], int lane) {
    int n = V / 2, o = 16;
#pragma unroll
    for (; n >= 1; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < V / 2; ++i)
            if (i < n) {
                const double keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
    }
    if (V == 16) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}

// r and 1 / r where r^2 leaves the range of fix64::root
__device__ __noinline__ double2 distance_library(double dx, double dy, double dz) {
    const double r = dev::julia_hypot3(dx, dy, dz);
    return make_double2(r, __ddiv_rn(1.0, r));
}

// negated unit normal and jacobian where the components leave the range of
// fix64::hypot3
struct Normal {
    double x, y, z, jac;
};
__device__ __noinline__ Normal normal_library(double n0, double n1, double n2) {
    const double jac = dev::julia_hypot3(n0, n1, n2);
    return Normal{__ddiv_rn(-n0, jac), __ddiv_rn(-n1, jac), __ddiv_rn(-n2, jac), jac};
}

// FLAT: three-node elements with linear shape functions, whose derivatives and
// so normal and jacobian are the same at every point.
//
// Bound by the FP64 pipe (62 cycles per operation and scheduler): 230
// operations per point when roots, divisions, sine, cosine and exponential came
// from the library and flat elements formed their normal at every point, some
// 50 now, with about 280 integer instructions beside them.  Flat elements, 1962
// nodes: 19.9 -> 4.2 ms (with a complex wavenumber 21.6 -> 4.8); 6-node elements,
// 2562 nodes: 36.0 -> 19.0 ms (interpolation and cross product stay in FP64 at every
// point; the hypot and divisions of the normal on the integer pipes with the same
// roundings were worth 27.4 -> 21.4, the zero derivatives left out 2.4 more).
template <int NS, int NP, bool CPLX_K, bool FLAT>
__global__ void __launch_bounds__(256)
nearfield_kernel(const int32_t *__restrict__ pairs, int pstride, int64_t npairs,
                 const double *__restrict__ table, int tstride, const __grid_constant__ RuleSet rs, bool coarse,
                 const double *__restrict__ coords, const int32_t *__restrict__ topo,
                 const double *__restrict__ tgt, double kre, double kim, int flags, double sign,
                 const int32_t *__restrict__ trig_tab, double2 *__restrict__ Fv, double2 *__restrict__ Gv) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const bool doF = flags & BIE_F, doG = flags & BIE_G;
    const dev::TrigFix trig{trig_tab};
    for (int64_t p = warp; p < npairs; p += nwarps) {
        const int32_t *pr = pairs + p * pstride;
        const int64_t i = pr[0];
        const int64_t e = pr[1];
        double X[3 * NS];
#pragma unroll
        for (int a = 0; a < NS; ++a) {
            const double *xa = coords + 3 * (int64_t)topo[(int64_t)NS * e + a];
            X[3 * a] = xa[0];
            X[3 * a + 1] = xa[1];
            X[3 * a + 2] = xa[2];
        }
        const double tx = tgt[3 * i], ty = tgt[3 * i + 1], tz = tgt[3 * i + 2];
        int64_t base;
        int Q;
        if (coarse) {
            base = rs.coarse_off;
            Q = rs.coarse_q;
        } else {
            const int c = dev::nearest_node<NS>(X, tx, ty, tz);
            base = rs.off[c];
            Q = rs.q[c];
        }
        // negated unit normal, jacobian / 4 pi
        double nx = 0, ny = 0, nz = 0, jac4 = 0;
        auto normal = [&](const double *P) {
            double tu[3] = {0, 0, 0}, tv[3] = {0, 0, 0};
#pragma unroll
            for (int a = 0; a < NS; ++a) {
                const double Ua = P[NS + a], Va = P[2 * NS + a];
                // (dN/du of the third corner and dN/dv of the second are zero)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    if (a != 2) tu[k] = a == 0 ? __dmul_rn(X[k], Ua) : __dadd_rn(tu[k], __dmul_rn(X[3 * a + k], Ua));
                    if (a != 1) tv[k] = a == 0 ? __dmul_rn(X[k], Va) : __dadd_rn(tv[k], __dmul_rn(X[3 * a + k], Va));
                }
            }
            const double n0 = __dsub_rn(__dmul_rn(tu[1], tv[2]), __dmul_rn(tu[2], tv[1]));
            const double n1 = __dsub_rn(__dmul_rn(tu[2], tv[0]), __dmul_rn(tu[0], tv[2]));
            const double n2 = __dsub_rn(__dmul_rn(tu[0], tv[1]), __dmul_rn(tu[1], tv[0]));
            // hypot and divisions with the roundings of the FP64 pipe
            double jac;
            if (fix64::hypot3(n0, n1, n2, jac)) {
                const fix64::Divisor d = fix64::divisor(jac);
                nx = fix64::divide(-n0, d);
                ny = fix64::divide(-n1, d);
                nz = fix64::divide(-n2, d);
            } else {
                const Normal l = normal_library(n0, n1, n2);
                jac = l.jac;
                nx = l.x;
                ny = l.y;
                nz = l.z;
            }
            jac4 = jac * kInv4Pi;
        };
        if (FLAT) normal(table + base * tstride);
        constexpr int V = NP <= 4 ? 16 : 32;
        double acc[V];   // fr, fi, gr, gi per node
#pragma unroll
        for (int a = 0; a < V; ++a) acc[a] = 0.0;
        for (int q = lane; q < Q; q += 32) {
            // The subdivided rules put points within 1e-6 element sizes of the
            // singular node, where x_q - t and n.(x_q - t) cancel (on flat elements
            // F is that rounding): the geometry is therefore evaluated with
            // separately rounded products and sums in the reference's order
            // (interpolation, cross product, Julia hypot for the jacobian, IEEE
            // division for the normal), so the result does not depend on FMA
            // contraction.  The functions of r only scale it.
            const double *P = table + (base + q) * tstride;
            double x[3] = {0, 0, 0};
#pragma unroll
            for (int a = 0; a < NS; ++a) {
                const double Na = P[a];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double m = __dmul_rn(X[3 * a + k], Na);
                    x[k] = a == 0 ? m : __dadd_rn(x[k], m);
                }
            }
            if (!FLAT) normal(P);
            const double jw = jac4 * P[3 * NS + NP];
            const double dx = __dsub_rn(x[0], tx), dy = __dsub_rn(x[1], ty), dz = __dsub_rn(x[2], tz);
            double rinv, rr;
            if (!fix64::root(dx * dx + dy * dy + dz * dz, rinv, rr)) {
                const double2 d = distance_library(dx, dy, dz);
                rr = d.x;
                rinv = d.y;
            }
            const double ai = kre * rr;
            double sn, cs;
            trig.sincos_of(ai, &sn, &cs);
            if (CPLX_K) {
                const double damp = trig.exp_minus(kim * rr);
                sn *= damp;
                cs *= damp;
            }
            const double wg = rinv * jw;
            const double *ph = P + 3 * NS;
            if (doF) {
                const double dn = __dadd_rn(__dadd_rn(__dmul_rn(nx, dx), __dmul_rn(ny, dy)), __dmul_rn(nz, dz));
                const double tq = dn * (wg * rinv) * rinv;
                double Fr, Fi;   // e^{ikr} (i k r - 1) tq
                if (CPLX_K) {
                    const double ar = -1.0 - kim * rr;
                    Fr = (cs * ar - sn * ai) * tq;
                    Fi = (cs * ai + sn * ar) * tq;
                } else {
                    Fr = -(sn * ai + cs) * tq;
                    Fi = (cs * ai - sn) * tq;
                }
#pragma unroll
                for (int a = 0; a < NP; ++a) {
                    acc[4 * a] += Fr * ph[a];
                    acc[4 * a + 1] += Fi * ph[a];
                }
            }
            if (doG) {
                const double Gr = cs * wg, Gi = sn * wg;
#pragma unroll
                for (int a = 0; a < NP; ++a) {
                    acc[4 * a + 2] += Gr * ph[a];
                    acc[4 * a + 3] += Gi * ph[a];
                }
            }
        }
        const double sum = warp_sums<V>(acc, lane);
        const int v = V == 32 ? lane : lane >> 1, a = v >> 2;
        if (v < 4 * NP && (V == 32 || !(lane & 1)) && ((v & 2) ? doG : doF)) {
            double2 *dst = ((v & 2) ? Gv : Fv) + pr[2 + a];
            atomicAdd((v & 1) ? &dst->y : &dst->x, sign * sum);
        }
    }
}

template <int NS, int NP>
void launch_ns_np(Ctx &c, const NearField &nf, double kre, double kim, int flags, bool coarse,
                  double sign, double *Fv, double *Gv) {
    RuleSet rs{};
    for (int r = 0; r < nf.nrules; ++r) {
        rs.off[r] = nf.rule_off[r];
        rs.q[r] = nf.rule_q[r];
    }
    rs.coarse_off = nf.coarse_off;
    rs.coarse_q = nf.coarse_q;
    const int64_t warps = std::min<int64_t>(nf.npairs, (int64_t)c.num_sms * 64);
    const unsigned blocks = (unsigned)std::max<int64_t>(1, (warps * 32 + 255) / 256);
    const bool cplx = kim != 0.0;
    cudaEvent_t t0 = c.timer_begin();
    constexpr bool kFlat = NS == 3;   // (three-node shape functions are linear)
    auto kern = cplx ? nearfield_kernel<NS, NP, true, kFlat> : nearfield_kernel<NS, NP, false, kFlat>;
    kern<<<blocks, 256, 0, c.stream>>>(nf.d_pairs, nf.pair_stride, nf.npairs, nf.d_table, nf.point_stride, rs, coarse,
                                       c.d_coords, c.d_topo, c.d_sources, kre, kim, flags, sign, c.d_xtrig,
                                       reinterpret_cast<double2 *>(Fv), reinterpret_cast<double2 *>(Gv));
    BIE_CUDA(cudaGetLastError());
    c.timer_end(t0);
    ++c.kernel_launches;
}

}  // namespace

void launch_nearfield(Ctx &c, const NearField &nf, double k_re, double k_im, int flags, bool coarse,
                      double sign, double *Fv, double *Gv) {
    if (nf.npairs == 0 || !(flags & (BIE_F | BIE_G))) return;
    if (c.NS == 3 && c.lay.NP == 3) launch_ns_np<3, 3>(c, nf, k_re, k_im, flags, coarse, sign, Fv, Gv);
    else if (c.NS == 6 && c.lay.NP == 6) launch_ns_np<6, 6>(c, nf, k_re, k_im, flags, coarse, sign, Fv, Gv);
    else if (c.NS == 6 && c.lay.NP == 3) launch_ns_np<6, 3>(c, nf, k_re, k_im, flags, coarse, sign, Fv, Gv);
    else fail(BIE_ERR_UNSUPPORTED, "near-field assembly for this element combination");
}

}  // namespace bie
