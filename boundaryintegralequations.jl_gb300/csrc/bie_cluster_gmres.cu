// One-launch restarted GMRES for the sparse near-field systems of the
// visco-thermal operator (the gmres(Gh, .) and gmres(Gv, .) calls of
// LossyGlobalOuter / LossyGlobalInner, src/3d/LossyGlobalMatrix.jl:26-37 and
// :179-197).
//
// Those systems are small (N or 3N rows, N = mesh nodes, a few to a few tens of
// non-zeros per row) and converge in a handful of Arnoldi steps, so the
// launch-per-operation form of the device GMRES (dot products, Gram-Schmidt
// updates, Givens steps, host checks) spends its time in launch latency.  Here
// one launch runs the whole solve:
//   * the rows are split into one contiguous range per CTA; the working vector
//     w and, where it fits, the Krylov basis V of the CTA's rows live in its
//     shared memory; the newest basis vector is also written to a global
//     vector, from which the sparse product gathers it; the iterate x is in
//     global memory (V too when it does not fit; all L2-resident here);
//   * every reduction (Gram-Schmidt coefficients, norms) is a per-warp pass
//     over the CTA's rows, a barrier, and a sum of the CTAs' partials in a
//     fixed order, so every CTA holds bit-identical coefficients and takes the
//     same branches;
//   * the Hessenberg column, Givens rotations, residual estimate and back
//     substitution run on one warp of each CTA on its own copy of the state, the
//     rotations while the other warps update w;
//   * a warp waits 62 cycles for each FP64 operation whatever its parallelism, so
//     the work is laid out for few operations in a row: real components, eight
//     lanes per matrix row, lanes shared between the columns of a dot product.
//     Solves of 2562 and 7686 rows, 3 steps, with a polling loop that reads the
//     error word seldom: 108 -> 74 us on average.
// Two synchronisation forms:
//   * grid (large systems): one CTA per SM, partials in global memory, a
//     grid barrier of this file (one monotonic arrival counter: barrier b
//     completes when it reaches (b + 1) x CTAs; release add, acquire polls)
//     whose waits are bounded: a wait that runs out sets an error word, which
//     makes every later barrier return at once, and the host reports the
//     error.  The launch is cooperative, so all CTAs are resident.  The
//     arithmetic is FP64 and this GPU's FP64 pipe is narrow, so the rows are
//     spread over all SMs;
//   * cluster (small systems): a 16-CTA (else 8-CTA) thread-block cluster,
//     partials read through distributed shared memory after hardware cluster
//     barriers, which every CTA reaches the same number of times.
// The algorithm is the device GMRES of bie_solver.cu (gmres_core): zero start,
// classical Gram-Schmidt with one re-orthogonalisation, complex Givens
// rotations (real cosine), restart after `restart` steps with the true
// residual, stop when |r| <= max(reltol |b|, abstol) or after maxiter steps.
// Every loop has a bound.
#include "bie_internal.h"
#include "bie_krylov.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

namespace cg = cooperative_groups;

namespace bie {

namespace {

constexpr int kMaxRestart = 48;        // longest restart cycle of the one-launch path
constexpr size_t kMaxSmem = 224 * 1024;
constexpr int kClusterThreads = 512;
constexpr int kGridThreads = 256;
constexpr unsigned kSpinLimit = 1u << 22;     // grid-barrier polls (a few seconds)

struct CgArgs {
    const int64_t *rp;
    const int32_t *cols;
    const double2 *val;
    const double2 *diag;   // may be null
    int64_t N;             // rows of one block
    int64_t n;             // nb * N
    const double2 *b;
    double2 *x;
    double2 *V;            // VS: the newest basis vector (n); else the basis, (m + 1) x n
    double2 *gpart;        // grid form: partials, 3 slots x (m + 2) columns x CTAs
    unsigned *bar;         // grid form: arrival counter (zero at launch)
    int *err;              // grid form: set when a barrier wait runs out
    int64_t rows_per;      // rows per CTA
    int m, maxiter;
    double reltol, abstol;
    bie_gmres_info *info;          // may be null
    unsigned long long *acc;       // [0] += 1 solve, [1] += iterations (may be null)
};

struct CgScalars {
    double res;     // |g_{j+1}| after the last step
    double na2, ia; // |a|^2 and 1 / |a| of the new column's last entry a
    double rh, in;  // 1 / h_{j+1,j}, 1 / sqrt(na2 + h_{j+1,j}^2)
    int done;       // converged or breakdown in this cycle
    int jdone;      // steps completed in this cycle
};

using namespace krylov;
// Threads of a CTA that share the partial sums: one warp per scheduler, since
// further warps only queue for its FP64 unit.
constexpr int kSumThreads = 128;

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_add_release(unsigned *p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Synchronisation over a thread-block cluster: partials in shared memory,
// read by the other CTAs through distributed shared memory.
template <int NT>
struct ClusterSync {
    static constexpr int kThreads = NT;
    cg::cluster_group cl;
    double2 *spart;   // shared: 3 slots x ps
    int ps;
    __device__ ClusterSync(const CgArgs &, double2 *spart_, int ps_) : cl(cg::this_cluster()), spart(spart_), ps(ps_) {}
    __device__ unsigned rank() const { return cl.block_rank(); }
    __device__ void sync() { cl.sync(); }
    // where this CTA writes column c of slot s (stride between columns)
    __device__ double2 *mine(int s) const { return spart + s * ps; }
    __device__ int stride() const { return 1; }
    // out[c] = sum over CTAs of their slot-s partial of column c (after sync)
    __device__ void gather(int s, int nc, double2 *out) {
        const int C = (int)cl.num_blocks(), L = 16;
        for (int q0 = threadIdx.x / 32 * (32 / L); q0 < 2 * nc; q0 += NT / L) {
            const int q = q0 + threadIdx.x % 32 / L, k = threadIdx.x % L;
            double v = 0.0;
            if (q < 2 * nc && k < C) v = comps(cl.map_shared_rank(spart + s * ps, (unsigned)k))[q];
            v = lane_sum(v, L);
            if (k == 0 && q < 2 * nc) comps(out)[q] = v;
        }
    }
    __device__ void finish() { cl.sync(); }   // no CTA leaves while another reads its shared memory
};

// Synchronisation over a cooperative grid: partials in global memory, a
// bounded counting barrier.  The CTA barrier before the release add makes the
// CTA's writes visible with it; the acquire poll and the CTA barrier after it
// order the CTA's later reads.
template <int NT>
struct GridSync {
    static constexpr int kThreads = NT;
    double2 *gpart;
    unsigned *count;
    int *err;
    int ps;
    unsigned nb, r, target;
    bool dead = false;   // thread 0: a wait ran out, here or elsewhere
    __device__ GridSync(const CgArgs &a, double2 *, int ps_)
        : gpart(a.gpart), count(a.bar), err(a.err), ps(ps_), nb(gridDim.x), r(blockIdx.x), target(0) {}
    __device__ unsigned rank() const { return r; }
    __device__ void sync() {
        target += nb;
        __syncthreads();
        if (threadIdx.x == 0 && !dead) {
            red_add_release(count, 1u);
            // (the error word only every 64 polls: reading it with each one doubles
            // the time between two looks at the counter)
            for (unsigned spins = 1; (int)(ld_acquire(count) - target) < 0; ++spins) {
                if (spins % 64 == 0 && (spins > kSpinLimit || ld_relaxed(err) != 0)) {
                    atomicExch(err, 1);
                    dead = true;
                    break;
                }
            }
        }
        __syncthreads();
    }
    __device__ double2 *mine(int s) const { return gpart + (size_t)s * ps * nb + r; }
    __device__ int stride() const { return (int)nb; }
    __device__ void gather(int s, int nc, double2 *out) {
        if (threadIdx.x >= kSumThreads) return;
        const double *base = comps(gpart + (size_t)s * ps * nb);
        const int L = lanes_per<kSumThreads>(nc), k = threadIdx.x % L;
        for (int q0 = 0; q0 < 2 * nc; q0 += kSumThreads / L) {
            const int q = q0 + threadIdx.x / L;
            double v = 0.0;
            if (q < 2 * nc) {
                const double *p = base + 2 * (size_t)(q >> 1) * nb + (q & 1);
#pragma unroll 8
                for (unsigned b = k; b < nb; b += L) v += __ldcg(p + 2 * b);
            }
            v = lane_sum(v, L);
            if (k == 0 && q < 2 * nc) comps(out)[q] = v;
        }
    }
    __device__ void finish() {}
};

// out(i, im, component im of (A s)[lo + i]) for the CTA's rows; s was written by
// other CTAs before the last barrier, so it is read through L2
template <int NT, class Out>
__device__ __forceinline__ void csr_rows(const CgArgs &a, const double2 *s, int64_t lo, int cnt, Out out) {
    const int lane = threadIdx.x & 31;
    const bool im = lane & 1;
    for (int r0 = threadIdx.x / 32 * 4; r0 < cnt; r0 += NT / 8) {
        const int i = r0 + (lane >> 3);
        const bool in = i < cnt;
        const int64_t blk = in ? (lo + i) / a.N : 0, r = lo + i - blk * a.N;
        double v = row_product<true>(a.rp, a.cols, a.val, s + blk * a.N, r, in, lane);
        if (in && (lane & 6) == 0) {
            if (a.diag) v = mul_step(v, __ldg(a.diag + r), __ldcg(s + lo + i), im);
            out(i, im, v);
        }
    }
}

// part[c * pst] = V[:, c]^H w over this CTA's rows, c < nc; column c of the CTA's
// rows starts at Vl + c * ld
__device__ __forceinline__ void local_multidot(const double2 *Vl, int64_t ld, int cnt, int nc, const double2 *w_s,
                                               double2 *part, int pst) {
    if (threadIdx.x >= kSumThreads) return;
    const int L = lanes_per<kSumThreads>(nc), lane = threadIdx.x % L;
    for (int q0 = 0; q0 < 2 * nc; q0 += kSumThreads / L) {
        const int q = q0 + threadIdx.x / L;
        double v = 0.0;
        if (q < 2 * nc) {
            const double2 *vc = Vl + (int64_t)(q >> 1) * ld;
#pragma unroll 4
            for (int i = lane; i < cnt; i += L) v = dot_step(v, vc[i], w_s[i], q & 1);
        }
        v = lane_sum(v, L);
        if (lane == 0 && q < 2 * nc) comps(part + (int64_t)(q >> 1) * pst)[q & 1] = v;
    }
}

// part[0] = |w|^2 over this CTA's rows, by the first warp
__device__ __forceinline__ void local_norm2(int cnt, const double2 *w_s, double2 *part) {
    if (threadIdx.x >= 32) return;
    double s = 0.0;
    for (int i = threadIdx.x; i < 2 * cnt; i += 32) s = fma(comps(w_s)[i], comps(w_s)[i], s);
    s = lane_sum(s, 32);
    if (threadIdx.x == 0) part[0] = make_double2(s, 0.0);
}

template <class Sync, bool VS>
__global__ void __launch_bounds__(Sync::kThreads, 1) csr_gmres_one_kernel(CgArgs a) {
    constexpr int NT = Sync::kThreads;
    const int m = a.m;
    const int64_t n = a.n;
    const int ps = m + 2;

    // shared memory: [VS: basis (m + 1) x rows_per], w (rows_per), three
    // partial slots (m + 2 each; cluster form), h1, h2, y (m + 2 each),
    // H ((m + 1) x m), g (m + 1), sn (m), cs (m), scalars
    extern __shared__ double2 smem[];
    double2 *V_s = smem;
    double2 *w_s = VS ? smem + (int64_t)(m + 1) * a.rows_per : smem;
    double2 *spart = w_s + a.rows_per;
    double2 *h1 = spart + 3 * ps;
    double2 *h2 = h1 + ps;
    double2 *y = h2 + ps;
    double2 *H = y + ps;
    double2 *g = H + (int64_t)(m + 1) * m;
    double2 *sn = g + (m + 1);
    double *cs = reinterpret_cast<double *>(sn + m);
    CgScalars *sc = reinterpret_cast<CgScalars *>(cs + m);

    Sync S(a, spart, ps);
    const int rank = (int)S.rank();
    const int lane = threadIdx.x & 31;
    const bool last = threadIdx.x >= NT - 32;   // the warp that keeps the Hessenberg system
    const int64_t lo0 = (int64_t)rank * a.rows_per;
    const int64_t lo = lo0 < n ? lo0 : n;
    const int64_t hi = lo + a.rows_per < n ? lo + a.rows_per : n;
    const int cnt = (int)(hi - lo);
    // this CTA's rows of basis column c: Vl + c * ldv
    double2 *Vl = VS ? V_s : a.V + lo;
    const int64_t ldv = VS ? a.rows_per : n;

    int slot = 0;
    // reduction into out[0..nc): this CTA's partials are in slot `s` already
    auto reduce = [&](int s, int nc, double2 *out) {
        S.sync();
        S.gather(s, nc, out);
        __syncthreads();
    };
    auto next_slot = [&]() {
        const int s = slot;
        slot = slot == 2 ? 0 : slot + 1;
        return s;
    };

    // |b|, x = 0, w = b
    for (int i = threadIdx.x; i < cnt; i += NT) {
        w_s[i] = a.b[lo + i];
        a.x[lo + i] = make_double2(0.0, 0.0);
    }
    __syncthreads();
    {
        const int s = next_slot();
        local_norm2(cnt, w_s, S.mine(s));
        reduce(s, 1, h1);
    }
    const double bnorm = sqrt(fmax(h1[0].x, 0.0));
    const double tol = fmax(a.reltol * bnorm, a.abstol);
    double beta = bnorm;
    int it = 0, restarts = 0;
    long long matvecs = 0;

    for (int cycle = 0; cycle <= a.maxiter; ++cycle) {
        if (cycle > 0) {
            // w = b - A x with the x of every CTA
            S.sync();
            csr_rows<NT>(a, a.x, lo, cnt, [&](int i, int im, double v) {
                comps(w_s)[2 * i + im] = comps(a.b)[2 * (lo + i) + im] - v;
            });
            ++matvecs;
            __syncthreads();
            const int s = next_slot();
            local_norm2(cnt, w_s, S.mine(s));
            reduce(s, 1, h1);
            beta = sqrt(fmax(h1[0].x, 0.0));
        }
        const int jmax = min(m, max(0, a.maxiter - it));
        if (beta <= tol || jmax == 0) break;

        // v_0 = w / beta; g = (beta, 0, ...)
        const double inv_beta = 1.0 / beta;
        for (int i = threadIdx.x; i < cnt; i += NT) {
            const double2 v = make_double2(w_s[i].x * inv_beta, w_s[i].y * inv_beta);
            Vl[i] = v;
            if (VS) a.V[lo + i] = v;
        }
        if (threadIdx.x == 0) {
            for (int k = 0; k <= m; ++k) g[k] = make_double2(0.0, 0.0);
            g[0] = make_double2(beta, 0.0);
            sc->res = beta;
            sc->done = 0;
            sc->jdone = 0;
        }
        for (int j = 0; j < jmax; ++j) {
            S.sync();   // v_j of every CTA is in global memory
            const double2 *vj = VS ? a.V : a.V + (int64_t)j * n;
            csr_rows<NT>(a, vj, lo, cnt, [&](int i, int im, double v) { comps(w_s)[2 * i + im] = v; });
            __syncthreads();
            // classical Gram-Schmidt, two passes
            for (int pass = 0; pass < 2; ++pass) {
                double2 *h = pass == 0 ? h1 : h2;
                const int s = next_slot();
                local_multidot(Vl, ldv, cnt, j + 1, w_s, S.mine(s), S.stride());
                reduce(s, j + 1, h);
                if (!last) {
                    for (int i = threadIdx.x; i < 2 * cnt; i += NT - 32) {
                        double v = 0.0;
#pragma unroll 4
                        for (int c = 0; c <= j; ++c) v = mul_step(v, Vl[(int64_t)c * ldv + (i >> 1)], h[c], i & 1);
                        comps(w_s)[i] -= v;
                    }
                } else if (pass == 1 && lane < 4) {
                    // meanwhile the earlier rotations of Hessenberg column j
                    double2 *col = H + (int64_t)j * (m + 1);
                    for (int k = lane; k <= j; k += 4) col[k] = make_double2(h1[k].x + h2[k].x, h1[k].y + h2[k].y);
                    __syncwarp(0xfu);
                    rotate_column(col, sn, cs, j, lane);
                    if (lane == 0) {
                        const double2 u = col[j];
                        sc->na2 = fma(u.x, u.x, u.y * u.y);
                        sc->ia = rsqrt(sc->na2);
                    }
                }
                __syncthreads();
            }
            {
                const int s = next_slot();
                local_norm2(cnt, w_s, S.mine(s));
                reduce(s, 1, y);
            }
            const double hn2 = fmax(y[0].x, 0.0);
            if (threadIdx.x == 0) sc->in = rsqrt(sc->na2 + hn2);
            if (threadIdx.x == 32) sc->rh = rsqrt(hn2);
            __syncthreads();
            Rotation rot{};
            if (!last) {
                // v_{j+1} = w / h_{j+1,j}
                const double inv_hn = hn2 > 0.0 ? sc->rh : 0.0;
                double *vn = comps(Vl + (int64_t)(j + 1) * ldv);
                for (int i = threadIdx.x; i < 2 * cnt; i += NT - 32) {
                    const double v = comps(w_s)[i] * inv_hn;
                    vn[i] = v;
                    // the global copy of v_j was last read by the products before
                    // this step's first reduction barrier
                    if (VS) comps(a.V + lo)[i] = v;
                }
            } else if (lane == 0) {
                rot = last_rotation(H[(int64_t)j * (m + 1) + j], sc->na2, sc->ia, hn2, sc->rh, sc->in);
                sc->res *= rot.q;   // (|g_{j+1}|: g_{j+1} was 0)
                sc->jdone = j + 1;
                sc->done = (sc->res <= tol || hn2 == 0.0) ? 1 : 0;
            }
            __syncthreads();
            const bool done = sc->done;
            if (last && lane == 0) {   // (read by this warp, or after a barrier)
                double2 *col = H + (int64_t)j * (m + 1);
                cs[j] = rot.c;
                sn[j] = rot.sn;
                col[j] = rot.r;
                col[j + 1] = make_double2(0.0, 0.0);
                const double2 gj = g[j], ug = cmul(cconj(rot.sn), gj);
                g[j] = make_double2(rot.c * gj.x, rot.c * gj.y);
                g[j + 1] = make_double2(-ug.x, -ug.y);
            }
            if (done) break;
        }
        // y = R^{-1} g; x += V y (this CTA's rows)
        __syncthreads();
        const int jd = sc->jdone;
        if (threadIdx.x < 32) {
            for (int k = lane; k < jd; k += 32) y[k] = g[k];
            __syncwarp();
            back_substitute(H, m + 1, jd, y, lane);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < 2 * cnt; i += NT) {
            double v = comps(a.x + lo)[i];
#pragma unroll 4
            for (int c = 0; c < jd; ++c) v = mul_step(v, Vl[(int64_t)c * ldv + (i >> 1)], y[c], i & 1);
            comps(a.x + lo)[i] = v;
        }
        it += jd;
        matvecs += jd;
        ++restarts;
    }
    if (rank == 0 && threadIdx.x == 0) {
        if (a.info) {
            bie_gmres_info o{};
            o.iterations = it;
            o.restarts = restarts;
            o.refinements = 0;
            o.converged = beta <= tol ? 1 : 0;
            o.matvecs = matvecs;
            o.residual_norm = beta;
            o.rhs_norm = bnorm;
            *a.info = o;
        }
        if (a.acc) {
            atomicAdd(a.acc, 1ull);
            atomicAdd(a.acc + 1, (unsigned long long)it);
        }
    }
    S.finish();
}

size_t smem_bytes(int64_t rows_per, int m, bool vs) {
    const size_t c2 = (size_t)rows_per * (vs ? m + 2 : 1) + 3 * (m + 2) + 3 * (m + 2) + (size_t)(m + 1) * m +
                      (m + 1) + m;
    return c2 * 16 + (size_t)m * 8 + sizeof(CgScalars) + 16;
}

// Whether kernel `kern` launches with `blocks` CTAs of `threads` threads and
// `smem` bytes each: as a cluster of `blocks` CTAs (cluster form), or all
// resident at once (grid form).  Cached per (kernel, device, smem, blocks).
// The kernel's dynamic shared-memory limit is raised once per device to the
// largest size this path launches with (kMaxSmem), so every cached answer
// stays launchable.
bool launch_fits(const void *kern, bool cluster, int device, int num_sms, size_t smem, int blocks, int threads) {
    static std::mutex mu;
    static std::map<std::tuple<const void *, int, size_t, int>, bool> cache;
    static std::map<std::pair<const void *, int>, bool> attrs_ok;
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_tuple(kern, device, smem, blocks);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    auto at_it = attrs_ok.find({kern, device});
    if (at_it == attrs_ok.end()) {
        bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) == cudaSuccess;
        if (cluster)
            ok = ok && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        at_it = attrs_ok.emplace(std::make_pair(kern, device), ok).first;
    }
    bool fits = false;
    if (at_it->second) {
        if (cluster) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(blocks);
            cfg.blockDim = dim3(threads);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = blocks;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int nclusters = 0;
            fits = cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) == cudaSuccess && nclusters > 0;
        } else {
            int per_sm = 0;
            fits = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) == cudaSuccess &&
                   (int64_t)per_sm * num_sms >= blocks;
        }
    }
    cudaGetLastError();
    cache[key] = fits;
    return fits;
}

struct Form {
    const void *kern;
    bool cluster, vs;
    int threads;
};

}  // namespace

bool csr_gmres_one_launch(Ctx &c, const CsrSystem &A, const double2 *b, double2 *x, const bie_gmres_opts &o,
                          int level, bie_gmres_info *d_info, unsigned long long *d_acc, int *d_err, int forms) {
    const int64_t n = A.N * A.nb;
    if (n <= 0 || c.capturing) return false;
    const int m = (int)std::max<int64_t>(1, std::min<int64_t>(o.restart > 0 ? o.restart : 20, n));
    if (m > kMaxRestart) return false;
    const int maxiter = o.maxiter > 0 ? o.maxiter : (int)std::min<int64_t>(n, INT32_MAX);
    // Launch forms in order of preference.  Systems of more than 2048 rows go
    // to the grid form (the FP64 work spread over up to one CTA per SM, 32 rows
    // or more per CTA), smaller ones to a cluster; the basis in shared memory
    // where it fits.  `forms` may restrict the choice to one of the two.
    const Form grid_vs{reinterpret_cast<const void *>(csr_gmres_one_kernel<GridSync<kGridThreads>, true>), false,
                       true, kGridThreads};
    const Form grid_g{reinterpret_cast<const void *>(csr_gmres_one_kernel<GridSync<kGridThreads>, false>), false,
                      false, kGridThreads};
    const Form cl_vs{reinterpret_cast<const void *>(csr_gmres_one_kernel<ClusterSync<kClusterThreads>, true>),
                     true, true, kClusterThreads};
    const Form cl_g{reinterpret_cast<const void *>(csr_gmres_one_kernel<ClusterSync<kClusterThreads>, false>),
                    true, false, kClusterThreads};
    std::vector<std::pair<Form, int>> cands;
    const bool grid_ok = d_err && forms != kOneLaunchCluster;
    if (grid_ok && (n > 2048 || forms == kOneLaunchGrid)) {
        const int P = (int)std::max<int64_t>(1, std::min<int64_t>(c.num_sms, (n + 31) / 32));
        cands = {{grid_vs, P}, {grid_g, P}};
    }
    if (forms != kOneLaunchGrid)
        for (const Form &f : {cl_vs, cl_g})
            for (const int cs : {16, 8}) cands.push_back({f, cs});
    Form form{};
    int P = 0;
    int64_t rows_per = 0;
    size_t smem = 0;
    for (const auto &cd : cands) {
        const int64_t rp = (n + cd.second - 1) / cd.second;
        const size_t sm = smem_bytes(rp, m, cd.first.vs);
        if (sm > kMaxSmem || !launch_fits(cd.first.kern, cd.first.cluster, c.device, c.num_sms, sm, cd.second,
                                          cd.first.threads))
            continue;
        form = cd.first;
        P = cd.second;
        rows_per = rp;
        smem = sm;
        break;
    }
    if (P == 0) return false;

    // workspace: basis (or its newest vector), grid partials, barrier words
    const int ws_slot = level == 0 ? kScratchSolver : kScratchSolverNested + 2 * (level - 1);
    const size_t vbytes = (size_t)(form.vs ? 1 : m + 1) * n * 16;
    const size_t pbytes = form.cluster ? 0 : (size_t)3 * (m + 2) * P * 16;
    char *ws = static_cast<char *>(c.scratch(ws_slot, vbytes + pbytes + 16));
    unsigned *bar = reinterpret_cast<unsigned *>(ws + vbytes + pbytes);
    if (!form.cluster) BIE_CUDA(cudaMemsetAsync(bar, 0, 8, c.stream));

    CgArgs a{};
    a.rp = A.rp;
    a.cols = A.cols;
    a.val = A.val;
    a.diag = A.diag;
    a.N = A.N;
    a.n = n;
    a.b = b;
    a.x = x;
    a.V = reinterpret_cast<double2 *>(ws);
    a.gpart = reinterpret_cast<double2 *>(ws + vbytes);
    a.bar = bar;
    a.err = d_err;
    a.rows_per = rows_per;
    a.m = m;
    a.maxiter = maxiter;
    a.reltol = o.reltol > 0 ? o.reltol : std::sqrt(2.220446049250313e-16);
    a.abstol = std::max(0.0, o.abstol);
    a.info = d_info;
    a.acc = d_acc;

    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(P);
    cfg.blockDim = dim3(form.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    if (form.cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = P;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void *args[] = {&a};
    BIE_CUDA(cudaLaunchKernelExC(&cfg, form.kern, args));
    ++c.kernel_launches;
    return true;
}

}  // namespace bie
