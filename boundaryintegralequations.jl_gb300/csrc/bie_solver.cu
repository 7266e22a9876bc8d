// K5: restarted GMRES on the device for  A x = b  with
//     A x = s (K x) + d .* x,
// K either a stored dense matrix (complex128 or complex64, column-major, the
// output of the assembly) or the matrix-free double-layer operator F.
// This replaces IterativeSolvers.gmres (v0.9) as called by the reference
// (test/3d/assembly_test.jl:38, examples/3d_pulsating_sphere.jl:44-50):
// same defaults (restart = min(20, N), reltol = sqrt(eps(Float64)), abstol 0,
// maxiter = N, x0 = 0) and the same stopping test ||r|| <= max(reltol ||b||,
// abstol) on the Arnoldi residual estimate.
//
// Arnoldi uses classical Gram-Schmidt with one reorthogonalisation pass
// (CGS2, the same numerical role as IterativeSolvers' default DGKS
// orthogonalisation); the small Hessenberg least-squares problem is solved with
// Givens rotations on the device (FP64).  Mixed-precision iterative refinement
// (opts->refine) runs the inner GMRES on the cheaper operator (complex64 dense
// copy or mixed matrix-free product) and forms the outer residual b - A x with
// the FP64 operator.
#include "bie_internal.h"
#include "bie_device.cuh"
#include "bie_fix64.cuh"
#include "bie_krylov.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace bie {

namespace {

constexpr int kT = 256;

// part[s n + i] = sum_j A[i + j n] x[j] (complex128) over the columns of slice
// blockIdx.y.
//
// The FP64 pipe would bound it at a fifth of the HBM rate (four FP64
// multiply-adds per 16 bytes at 2 lanes per clock and SM: 1.5 TB/s, 239 us at
// 4842 nodes), so the products run on the integer pipe.  Each component of x
// becomes an integer of 57 bits against its element's exponent, each matrix
// component one of 56 bits against E - (exponent of x), where E is the exponent
// of the row's largest product so far (raised when a larger one comes).  In
// limbs of radix 2^29 the products of the low limbs, which are left out, are below
// 2^-56 of that largest product; high x high and the two cross products are
// one IMAD.WIDE each and summed exactly, and every 64 columns the sums are
// added to the row's FP64 sum.  A block with an infinity, a NaN or only products
// near the subnormals (where a zero's hidden bit would count) is summed in FP64
// instead.
//
// Measured: 2562 nodes 92 -> 36 us, 4842 264 -> 94 us (4.0 TB/s), 10242
// 1193 -> 397 us (4.2 TB/s); the integer issue slots (about 110 per entry and
// warp) bound it now.  Error against extended precision, 5 to 2200 columns,
// entries and vectors spread over up to 300 decades: 0.7 to 1.01 times the FP64
// sum's.  Four columns are loaded ahead of the four in work (eight together
// without that: 38 / 103 / 430 us); two or four blocks per SM take 2 to 17 % longer.
constexpr int kGemvRadix = 29;
constexpr int kGemvMask = (1 << kGemvRadix) - 1;
__device__ __forceinline__ int biased_exponent(double a) { return (__double2hiint(a) >> 20) & 0x7ff; }
// a against the biased exponent E: a 2^(57 - (E - 1022)), truncated, as limbs
// (E at or above a's own exponent)
__device__ __forceinline__ fix64::Limb gemv_entry(double a, int ex, int E) {
    const int hi = __double2hiint(a);
    // (the hidden bit of a subnormal is shifted out)
    const long long m = fix64::make64((hi & 0xfffff) | 0x100000, (unsigned)__double2loint(a));
    const long long v = fix64::shift_right(m << 4, E - ex);
    const int s = hi >> 31;
    return fix64::Limb{((int)(v >> kGemvRadix) ^ s) - s, (((int)v & kGemvMask) ^ s) - s};
}
// (h + l 2^-29) 2^20 with one rounding; 0 <= l < 2^29
__device__ __forceinline__ double gemv_sum(long long h, long long l) {
    const long long low = (long long)((unsigned long long)(unsigned)h << 20) + (l >> (kGemvRadix - 20));
    return fma((double)(int)(h >> 32), 0x1p52, (double)low);
}
// x as limbs with a balanced low one
__device__ __forceinline__ fix64::Limb gemv_operand(long long v) {
    const int h = (int)((v + (1LL << (kGemvRadix - 1))) >> kGemvRadix);
    return fix64::Limb{h, (int)(v - ((long long)h << kGemvRadix))};
}

__global__ void __launch_bounds__(kT, 3)
dense_gemv_kernel(const double2 *__restrict__ A, int64_t n, const double2 *__restrict__ x,
                  double2 *__restrict__ part, int S, const int *__restrict__ stop) {
    if (stop && *stop) return;
    const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
    const int s = blockIdx.y;
    const int64_t j0 = (int64_t)s * n / S, j1 = (int64_t)(s + 1) * n / S;
    __shared__ double2 xs[kT];
    __shared__ int4 xf[kT];        // Re, Im limbs
    __shared__ __align__(16) int xe[kT];   // exponents
    __shared__ int s_max[kT / 32];
    constexpr int kRun = 4;              // columns loaded together, one run ahead
    constexpr int kBlock = 64;           // columns between additions to the FP64 sum
    double re = 0, im = 0;
    int E = 0;                           // exponent of the row's products (doubly biased)
    for (int64_t jb = j0; jb < j1; jb += kT) {
        const int nb = (int)min((int64_t)kT, j1 - jb);
        __syncthreads();
        {
            double2 v = make_double2(0.0, 0.0);
            if (threadIdx.x < nb) v = x[jb + threadIdx.x];
            xs[threadIdx.x] = v;
            const int ex = max(1, max(biased_exponent(v.x), biased_exponent(v.y)));
            xe[threadIdx.x] = ex;
            const int sc = 56 + 1022 - ex;
            const fix64::Limb a = gemv_operand(__double2ll_rn(ldexp(v.x, sc))),
                              b = gemv_operand(__double2ll_rn(ldexp(v.y, sc)));
            xf[threadIdx.x] = make_int4(a.h, a.l, b.h, b.l);
            int mx = ex;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
        }
        __syncthreads();
        if (i >= n) continue;
        int xmax = s_max[0];
#pragma unroll
        for (int k = 1; k < kT / 32; ++k) xmax = max(xmax, s_max[k]);
        const double2 *col = A + jb * n + i;
        // (past the chunk: its last column again, against x = 0)
        double2 next[kRun];
#pragma unroll
        for (int j = 0; j < kRun; ++j) next[j] = __ldcs(col + (int64_t)min(j, nb - 1) * n);
        for (int jc = 0; jc < nb; jc += kBlock) {
            const int ne = min(nb, jc + kBlock);
            long long hr = 0, lr = 0, hm = 0, lm = 0;   // sums in units 2^58 and 2^29
            int amax = 0;
            for (int j8 = jc; j8 < ne; j8 += kRun) {
                double2 a[kRun];
                int er[kRun], em[kRun], ex[kRun], top = 0;
#pragma unroll
                for (int j = 0; j < kRun; j += 4) {
                    const int4 e = *reinterpret_cast<const int4 *>(xe + j8 + j);
                    ex[j] = e.x;
                    ex[j + 1] = e.y;
                    ex[j + 2] = e.z;
                    ex[j + 3] = e.w;
                }
#pragma unroll
                for (int j = 0; j < kRun; ++j) {
                    a[j] = next[j];
                    next[j] = __ldcs(col + (int64_t)min(j8 + kRun + j, nb - 1) * n);
                }
#pragma unroll
                for (int j = 0; j < kRun; ++j) {
                    er[j] = biased_exponent(a[j].x);
                    em[j] = biased_exponent(a[j].y);
                    const int t = max(er[j], em[j]);
                    amax = max(amax, t);
                    top = max(top, t + ex[j]);
                }
                if (top > E) {   // a larger product: the sums so far move to its exponent
                    const int d = min(top - E, 127);
                    const __int128 tr = (((__int128)hr << kGemvRadix) + lr) >> d;
                    const __int128 tm = (((__int128)hm << kGemvRadix) + lm) >> d;
                    hr = (long long)(tr >> kGemvRadix);
                    lr = (long long)((int)tr & kGemvMask);
                    hm = (long long)(tm >> kGemvRadix);
                    lm = (long long)((int)tm & kGemvMask);
                    E = top;
                }
#pragma unroll
                for (int j = 0; j < kRun; ++j) {
                    const int Ej = E - ex[j];
                    const fix64::Limb ar = gemv_entry(a[j].x, er[j], Ej), ai = gemv_entry(a[j].y, em[j], Ej);
                    const int4 v = xf[j8 + j];
                    const fix64::Limb xr{v.x, v.y}, xi{v.z, v.w}, xn{-v.z, -v.w};
                    hr = fix64::high(fix64::high(hr, ar, xr), ai, xn);
                    lr = fix64::cross(fix64::cross(lr, ar, xr), ai, xn);
                    hm = fix64::high(fix64::high(hm, ar, xi), ai, xr);
                    lm = fix64::cross(fix64::cross(lm, ar, xi), ai, xr);
                }
                hr += lr >> kGemvRadix;
                lr = (long long)((int)lr & kGemvMask);
                hm += lm >> kGemvRadix;
                lm = (long long)((int)lm & kGemvMask);
            }
            if (amax < 0x7ff && xmax < 0x7ff && E > xmax + 64) {
                const int k = E - 2 * 1022 - 113 + 2 * kGemvRadix - 20;
                re += ldexp(gemv_sum(hr, lr), k);
                im += ldexp(gemv_sum(hm, lm), k);
            } else {
                for (int j = jc; j < ne; ++j) {
                    const double2 a = col[(int64_t)j * n], v = xs[j];
                    re += a.x * v.x - a.y * v.y;
                    im += a.x * v.y + a.y * v.x;
                }
                E = 0;
            }
        }
    }
    if (i < n) part[(int64_t)s * n + i] = make_double2(re, im);
}

// Complex64 matrix times complex128 vector on the FP32 pipe, for the column
// slice of blockIdx.y.  On GB300 the FP64 pipe cannot keep up with HBM even for
// a matrix-vector product, so the products run in FP32: the vector is rounded
// to FP32, every block of kFold columns is summed with plain FP32 FMAs and the
// block sums are carried in double-float (TwoSum).  The product then has a
// relative error of a few FP32 roundings (~1e-7) — the size of the complex64
// rounding of the stored matrix itself — at 8 FMAs per 16-byte load, which
// keeps the kernel on the HBM roofline.  Each thread handles two consecutive
// rows (one 16-byte load per column).
constexpr int kFold = 16;

__device__ __forceinline__ void df_fold(dev::df &acc, float s) {
    const dev::df t = dev::two_sum(acc.hi, s);
    acc = dev::fast_two_sum(t.hi, __fadd_rn(t.lo, acc.lo));
}

// The same product to ~1e-14 relative (the residuals of refinement and the
// right-hand sides): the vector is split into double-float (x = hi + lo),
// a * hi is formed exactly (TwoProduct), a * lo is added to its error term and
// every sum is carried in double-float (TwoSum).  About 14 instructions per
// real multiply-add, so issue-bound at roughly half the HBM rate.
__global__ void __launch_bounds__(kT)
dense_gemv_c64_exact_kernel(const float4 *__restrict__ A2, int64_t n, const double2 *__restrict__ x,
                            double2 *__restrict__ part, int S, const int *__restrict__ stop) {
    if (stop && *stop) return;
    const int64_t r2 = (int64_t)blockIdx.x * kT + threadIdx.x;   // row pair index
    const int64_t i0 = 2 * r2;
    const int s = blockIdx.y;
    const int64_t j0 = (int64_t)s * n / S, j1 = (int64_t)(s + 1) * n / S;
    __shared__ float4 xs[kT];   // (re hi, re lo, im hi, im lo)
    dev::df yr0 = {0.f, 0.f}, yi0 = {0.f, 0.f}, yr1 = {0.f, 0.f}, yi1 = {0.f, 0.f};
    const int64_t ld2 = n / 2;  // float4 per column (n even)
    auto mac = [](dev::df &acc, float av, float xh, float xl) {
        const float p = av * xh;
        float e = __fmaf_rn(av, xh, -p);
        e = __fmaf_rn(av, xl, e);
        const dev::df t = dev::two_sum(acc.hi, p);
        acc = dev::fast_two_sum(t.hi, __fadd_rn(__fadd_rn(t.lo, e), acc.lo));
    };
    for (int64_t jb = j0; jb < j1; jb += kT) {
        const int nb = (int)min((int64_t)kT, j1 - jb);
        __syncthreads();
        if (threadIdx.x < nb) {
            const double2 v = x[jb + threadIdx.x];
            const dev::df re = dev::df_from_double(v.x), im = dev::df_from_double(v.y);
            xs[threadIdx.x] = make_float4(re.hi, re.lo, im.hi, im.lo);
        }
        __syncthreads();
        if (i0 < n) {
            const float4 *col = A2 + jb * ld2 + r2;
#pragma unroll 4
            for (int j = 0; j < nb; ++j) {
                const float4 a = col[(int64_t)j * ld2];   // (re0, im0, re1, im1)
                const float4 xv = xs[j];
                mac(yr0, a.x, xv.x, xv.y);
                mac(yr0, -a.y, xv.z, xv.w);
                mac(yi0, a.x, xv.z, xv.w);
                mac(yi0, a.y, xv.x, xv.y);
                mac(yr1, a.z, xv.x, xv.y);
                mac(yr1, -a.w, xv.z, xv.w);
                mac(yi1, a.z, xv.z, xv.w);
                mac(yi1, a.w, xv.x, xv.y);
            }
        }
    }
    if (i0 < n) {
        part[(int64_t)s * n + i0] = make_double2(dev::f2d(yr0.hi) + dev::f2d(yr0.lo),
                                                 dev::f2d(yi0.hi) + dev::f2d(yi0.lo));
        if (i0 + 1 < n)
            part[(int64_t)s * n + i0 + 1] = make_double2(dev::f2d(yr1.hi) + dev::f2d(yr1.lo),
                                                         dev::f2d(yi1.hi) + dev::f2d(yi1.lo));
    }
}

// Odd n, exact form: one row per thread, 8-byte loads.
__global__ void __launch_bounds__(kT)
dense_gemv_c64_rows_exact_kernel(const float2 *__restrict__ A, int64_t n, const double2 *__restrict__ x,
                                 double2 *__restrict__ part, int S, const int *__restrict__ stop) {
    if (stop && *stop) return;
    const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
    const int s = blockIdx.y;
    const int64_t j0 = (int64_t)s * n / S, j1 = (int64_t)(s + 1) * n / S;
    __shared__ float4 xs[kT];
    dev::df yr = {0.f, 0.f}, yi = {0.f, 0.f};
    auto mac = [](dev::df &acc, float av, float xh, float xl) {
        const float p = av * xh;
        float e = __fmaf_rn(av, xh, -p);
        e = __fmaf_rn(av, xl, e);
        const dev::df t = dev::two_sum(acc.hi, p);
        acc = dev::fast_two_sum(t.hi, __fadd_rn(__fadd_rn(t.lo, e), acc.lo));
    };
    for (int64_t jb = j0; jb < j1; jb += kT) {
        const int nb = (int)min((int64_t)kT, j1 - jb);
        __syncthreads();
        if (threadIdx.x < nb) {
            const double2 v = x[jb + threadIdx.x];
            const dev::df re = dev::df_from_double(v.x), im = dev::df_from_double(v.y);
            xs[threadIdx.x] = make_float4(re.hi, re.lo, im.hi, im.lo);
        }
        __syncthreads();
        if (i < n) {
            const float2 *col = A + jb * n + i;
            for (int j = 0; j < nb; ++j) {
                const float2 a = col[(int64_t)j * n];
                const float4 xv = xs[j];
                mac(yr, a.x, xv.x, xv.y);
                mac(yr, -a.y, xv.z, xv.w);
                mac(yi, a.x, xv.z, xv.w);
                mac(yi, a.y, xv.x, xv.y);
            }
        }
    }
    if (i < n)
        part[(int64_t)s * n + i] = make_double2(dev::f2d(yr.hi) + dev::f2d(yr.lo),
                                                dev::f2d(yi.hi) + dev::f2d(yi.lo));
}

__global__ void __launch_bounds__(kT)
dense_gemv_c64_kernel(const float4 *__restrict__ A2, int64_t n, const double2 *__restrict__ x,
                      double2 *__restrict__ part, int S, const int *__restrict__ stop) {
    if (stop && *stop) return;
    const int64_t r2 = (int64_t)blockIdx.x * kT + threadIdx.x;   // row pair index
    const int64_t i0 = 2 * r2;
    const int s = blockIdx.y;
    const int64_t j0 = (int64_t)s * n / S, j1 = (int64_t)(s + 1) * n / S;
    __shared__ float2 xs[kT];
    dev::df yr0 = {0.f, 0.f}, yi0 = {0.f, 0.f}, yr1 = {0.f, 0.f}, yi1 = {0.f, 0.f};
    const int64_t ld2 = n / 2;  // float4 per column (n even)
    for (int64_t jb = j0; jb < j1; jb += kT) {
        const int nb = (int)min((int64_t)kT, j1 - jb);
        __syncthreads();
        if (threadIdx.x < nb) {
            const double2 v = x[jb + threadIdx.x];
            xs[threadIdx.x] = make_float2((float)v.x, (float)v.y);
        }
        __syncthreads();
        if (i0 < n) {
            const float4 *col = A2 + jb * ld2 + r2;
            for (int jf = 0; jf < nb; jf += kFold) {
                const int ne = min(kFold, nb - jf);
                float sr0 = 0.f, si0 = 0.f, sr1 = 0.f, si1 = 0.f;
                if (ne == kFold) {
#pragma unroll
                    for (int j = 0; j < kFold; ++j) {
                        const float4 a = col[(int64_t)(jf + j) * ld2];   // (re0, im0, re1, im1)
                        const float2 xv = xs[jf + j];
                        sr0 = __fmaf_rn(a.x, xv.x, sr0);
                        sr0 = __fmaf_rn(-a.y, xv.y, sr0);
                        si0 = __fmaf_rn(a.x, xv.y, si0);
                        si0 = __fmaf_rn(a.y, xv.x, si0);
                        sr1 = __fmaf_rn(a.z, xv.x, sr1);
                        sr1 = __fmaf_rn(-a.w, xv.y, sr1);
                        si1 = __fmaf_rn(a.z, xv.y, si1);
                        si1 = __fmaf_rn(a.w, xv.x, si1);
                    }
                } else {
                    for (int j = 0; j < ne; ++j) {
                        const float4 a = col[(int64_t)(jf + j) * ld2];
                        const float2 xv = xs[jf + j];
                        sr0 = __fmaf_rn(a.x, xv.x, sr0);
                        sr0 = __fmaf_rn(-a.y, xv.y, sr0);
                        si0 = __fmaf_rn(a.x, xv.y, si0);
                        si0 = __fmaf_rn(a.y, xv.x, si0);
                        sr1 = __fmaf_rn(a.z, xv.x, sr1);
                        sr1 = __fmaf_rn(-a.w, xv.y, sr1);
                        si1 = __fmaf_rn(a.z, xv.y, si1);
                        si1 = __fmaf_rn(a.w, xv.x, si1);
                    }
                }
                df_fold(yr0, sr0);
                df_fold(yi0, si0);
                df_fold(yr1, sr1);
                df_fold(yi1, si1);
            }
        }
    }
    if (i0 < n) {
        part[(int64_t)s * n + i0] = make_double2(dev::f2d(yr0.hi) + dev::f2d(yr0.lo),
                                                 dev::f2d(yi0.hi) + dev::f2d(yi0.lo));
        if (i0 + 1 < n)
            part[(int64_t)s * n + i0 + 1] = make_double2(dev::f2d(yr1.hi) + dev::f2d(yr1.lo),
                                                         dev::f2d(yi1.hi) + dev::f2d(yi1.lo));
    }
}

// Same product for odd n: one row per thread, 8-byte loads.
__global__ void __launch_bounds__(kT)
dense_gemv_c64_rows_kernel(const float2 *__restrict__ A, int64_t n, const double2 *__restrict__ x,
                           double2 *__restrict__ part, int S, const int *__restrict__ stop) {
    if (stop && *stop) return;
    const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
    const int s = blockIdx.y;
    const int64_t j0 = (int64_t)s * n / S, j1 = (int64_t)(s + 1) * n / S;
    __shared__ float2 xs[kT];
    dev::df yr = {0.f, 0.f}, yi = {0.f, 0.f};
    for (int64_t jb = j0; jb < j1; jb += kT) {
        const int nb = (int)min((int64_t)kT, j1 - jb);
        __syncthreads();
        if (threadIdx.x < nb) {
            const double2 v = x[jb + threadIdx.x];
            xs[threadIdx.x] = make_float2((float)v.x, (float)v.y);
        }
        __syncthreads();
        if (i < n) {
            const float2 *col = A + jb * n + i;
            for (int jf = 0; jf < nb; jf += kFold) {
                const int ne = min(kFold, nb - jf);
                float sr = 0.f, si = 0.f;
                for (int j = 0; j < ne; ++j) {
                    const float2 a = col[(int64_t)(jf + j) * n];
                    const float2 xv = xs[jf + j];
                    sr = __fmaf_rn(a.x, xv.x, sr);
                    sr = __fmaf_rn(-a.y, xv.y, sr);
                    si = __fmaf_rn(a.x, xv.y, si);
                    si = __fmaf_rn(a.y, xv.x, si);
                }
                df_fold(yr, sr);
                df_fold(yi, si);
            }
        }
    }
    if (i < n)
        part[(int64_t)s * n + i] = make_double2(dev::f2d(yr.hi) + dev::f2d(yr.lo),
                                                dev::f2d(yi.hi) + dev::f2d(yi.lo));
}

// ---- vector work of an Arnoldi step -------------------------------------------
// Between two products a step sums the product's slices, runs two Gram-Schmidt
// passes over the basis and normalises.  The vectors are short (77 KB at 4842
// nodes) and live in L2, so launches and the FP64 pipe bound them: a warp waits
// 62 cycles for each FP64 operation whatever its parallelism (measured; 16 cycles
// per warp operation and SM), and a launch costs about 2 us.  The step is four
// launches: each block owns a range of rows, keeps them through a launch, and
// takes for itself the sums of the partial sums that the launch before left per
// block (152 blocks at most), instead of a launch for each.  Threads work
// on real components, not complex numbers: half the operations in a row for each
// warp, and a warp per scheduler is enough to keep the pipe busy.
// 2562 nodes, 8 to 13 columns, 64 slices: 26 us a step in 4 launches; with one
// launch per sum, update and rotation 75 us in 7.  Solves of 8 wavenumbers (refined,
// with a sensitivity probe) 13.8 -> 7.6 ms.
constexpr int kRedBlocks = 152;   // most blocks of a vector kernel: one per SM
constexpr int kHs = 32;           // columns whose sums a block takes itself
constexpr int kVT = 128;          // threads where a block has few rows,
constexpr int kVTLong = 512;      // ... and many
constexpr int kLongRows = 128;
struct RowSplit {
    int64_t rows;   // per block, a multiple of 32
    int nb;
};
inline RowSplit row_split(int64_t n) {
    const int64_t rows = 32 * std::max<int64_t>(1, (n + 32 * kRedBlocks - 1) / (32 * kRedBlocks));
    return RowSplit{rows, (int)((n + rows - 1) / rows)};
}
using namespace krylov;

// done(i, sum over the groups g of term(i, g), the same of the row's other
// component) for the components i of rows r0 .. r1; two groups share the terms
// where the rows are few
template <int T>
constexpr int kGroups = T == kVT ? 2 : 1;
template <int T, typename Term, typename Done>
__device__ __forceinline__ void over_rows(int64_t r0, int64_t r1, double *red, Term term, Done done) {
    constexpr int G = kGroups<T>, RC = T / G;
    const int lane = threadIdx.x % RC, g = threadIdx.x / RC;
    for (int64_t base = 2 * r0; base < 2 * r1; base += RC) {
        const int64_t i = base + lane;
        double acc = i < 2 * r1 ? term(i, g) : 0.0;
        if (G > 1) {
            __syncthreads();
            if (g > 0) red[lane] = acc;
            __syncthreads();
            if (g == 0) acc += red[lane];
        }
        const double other = __shfl_xor_sync(0xffffffffu, acc, 1);
        if (g == 0 && i < 2 * r1) done(i, acc, other);
    }
}

// partial[c nb + block] = sum over rows r0 .. r1 of conj(V[:, c]) w
template <int T>
__device__ __forceinline__ void block_dots(const double2 *__restrict__ V, int64_t ldv, int ncol, const double2 *w,
                                           int64_t r0, int64_t r1, double2 *__restrict__ partial, int nb) {
    const int L = lanes_per<T>(ncol), lane = threadIdx.x % L;
    for (int q0 = 0; q0 < 2 * ncol; q0 += T / L) {
        const int q = q0 + threadIdx.x / L, c = q >> 1;
        const bool im = q & 1;
        double s = 0;
        if (q < 2 * ncol) {
            const double2 *v = V + (int64_t)c * ldv;
#pragma unroll 8
            for (int64_t i = r0 + lane; i < r1; i += L) {
                s = dot_step(s, v[i], w[i], im);
            }
        }
        s = lane_sum(s, L);
        if (lane == 0 && q < 2 * ncol) comps(partial)[2 * ((int64_t)c * nb + blockIdx.x) + (q & 1)] = s;
    }
}
// h[c] = sum of column c's nb partial sums, by the whole block
template <int T>
__device__ __forceinline__ void block_sums(const double2 *__restrict__ partial, int nb, int ncol, double2 *h) {
    const int L = lanes_per<T>(ncol), lane = threadIdx.x % L;
    for (int q0 = 0; q0 < 2 * ncol; q0 += T / L) {
        const int q = q0 + threadIdx.x / L;
        double s = 0;
        if (q < 2 * ncol) {
            const double *p = comps(partial) + 2 * (int64_t)(q >> 1) * nb + (q & 1);
#pragma unroll 16
            for (int b = lane; b < nb; b += L) s += p[2 * b];
        }
        s = lane_sum(s, L);
        if (lane == 0 && q < 2 * ncol) comps(h)[q] = s;
    }
}
// sum of the squares of one value per thread -> partial[block]
template <int T>
__device__ __forceinline__ void block_norm(double s, double *red, double *__restrict__ partial) {
    s = lane_sum(s, 32);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = red[0];
        for (int k = 1; k < T / 32; ++k) t += red[k];
        partial[blockIdx.x] = t;
    }
}
// the squared norm from block_norm's partial sums, in every thread
__device__ __forceinline__ double block_norm_value(const double *__restrict__ partial, int nb, double *red) {
    if (threadIdx.x < 32) {
        double s = 0;
#pragma unroll
        for (int k = 0; k <= kRedBlocks / 32; ++k) {
            const int b = threadIdx.x + k * 32;
            if (k * 32 < nb) s += b < nb ? partial[b] : 0.0;
        }
        s = lane_sum(s, 32);
        if (threadIdx.x == 0) red[0] = s;
    }
    __syncthreads();
    return fmax(red[0], 0.0);
}

// A product that is still in slices: y = sc sum_s part[s n + i] + d .* x (d may
// be null; part may be y if S == 1); S == 0: y already holds it.
struct Sliced {
    const double2 *part = nullptr;
    int S = 0;
    double2 sc = {1.0, 0.0};
    const double2 *d = nullptr, *x = nullptr;
};

// y = the product (or rhs - product, or rhs where *zero), then what the next
// launch needs: ncol > 0 the partial dot products with V, ncol < 0 the partial
// squared norms.
template <int T>
__global__ void __launch_bounds__(T)
gm_product_kernel(Sliced p, int64_t n, int64_t rows, double2 *y, const double2 *__restrict__ rhs,
                  const int *__restrict__ zero, const double2 *__restrict__ V, int ncol, double2 *__restrict__ dots,
                  double *__restrict__ norms, const int *__restrict__ stop) {
    if (stop && *stop) return;
    __shared__ double red[T];
    const int64_t r0 = (int64_t)blockIdx.x * rows, r1 = min(n, r0 + rows);
    double nrm = 0;
    const bool skip = zero && *zero;
    if (p.S > 0 || rhs || ncol < 0) {
        over_rows<T>(r0, r1, red,
            [&](int64_t i, int g) {
                double s = 0;
                if (skip) return s;
#pragma unroll 16
                for (int k = g; k < p.S; k += kGroups<T>) s += comps(p.part)[2 * (int64_t)k * n + i];
                return s;
            },
            [&](int64_t i, double s, double o) {
                const bool im = i & 1;
                double v;
                if (skip) {
                    v = 0;
                } else if (p.S == 0) {
                    v = comps(y)[i];
                } else {
                    v = fma(im ? p.sc.y : -p.sc.y, o, p.sc.x * s);
                    if (p.d) v = mul_step(v, p.d[i >> 1], p.x[i >> 1], im);
                }
                if (rhs) v = comps(rhs)[i] - v;
                if (p.S > 0 || rhs) comps(y)[i] = v;
                nrm = fma(v, v, nrm);
            });
    }
    if (ncol < 0) block_norm<T>(nrm, red, norms);
    if (ncol > 0) {
        __syncthreads();
        block_dots<T>(V, n, ncol, y, r0, r1, dots, gridDim.x);
    }
}

// out[c] = sum of column c's partial sums, one warp per column (bases of more
// than kHs columns, where each block's own sums would cost more than a launch)
__global__ void __launch_bounds__(kT)
sum_partials_kernel(const double2 *__restrict__ partial, int nb, int ncol, double2 *__restrict__ out,
                    const int *__restrict__ stop) {
    if (stop && *stop) return;
    const int c = blockIdx.x * (kT / 32) + threadIdx.x / 32;
    double re = 0, im = 0;
    if (c < ncol)
        for (int b = threadIdx.x & 31; b < nb; b += 32) {
            re += partial[(int64_t)c * nb + b].x;
            im += partial[(int64_t)c * nb + b].y;
        }
    re = lane_sum(re, 32);
    im = lane_sum(im, 32);
    if ((threadIdx.x & 31) == 0 && c < ncol) out[c] = make_double2(re, im);
}

// ---- device-resident Arnoldi state (one GMRES cycle without host round trips)
// Layout in one device block: H (m+1) x m, g (m+1), sn (m), h1 (m+1), h2 (m+1),
// y (m) complex; cs (m) real; scalars.
struct GmScalars {
    double beta;       // residual norm at the start of the cycle
    double res;        // |g_{j+1}| after the last step
    double tol;
    int done;          // 1: converged, breakdown or jmax steps; later kernels of the cycle skip
    int start_ok;      // 1: the starting residual already met the tolerance
    int jdone;         // Arnoldi steps completed in this cycle
    int jlast;         // ... in the cycle before
    int jmax;          // ... at most
};
struct GmState {
    double2 *H, *g, *sn, *h1, *h2, *y;
    double *cs;
    GmScalars *s;
    int m;
};

// out = a w over the block's rows
__device__ __forceinline__ void scale_rows(const double2 *__restrict__ w, double a, int64_t n, int64_t rows,
                                           double2 *__restrict__ out) {
    const int64_t r0 = (int64_t)blockIdx.x * rows, r1 = min(n, r0 + rows);
#pragma unroll 4
    for (int64_t i = 2 * r0 + threadIdx.x; i < 2 * r1; i += kVT) comps(out)[i] = a * comps(w)[i];
}

// state at the start of a cycle: g = (beta, 0, ...), done = beta <= tol
__device__ __forceinline__ void gm_begin(const GmState &st, double beta, double tol, int jmax) {
    GmScalars &s = *st.s;
    for (int k = threadIdx.x; k <= st.m; k += kVT) st.g[k] = make_double2(k ? 0.0 : beta, 0.0);
    if (threadIdx.x > 0) return;
    s.tol = tol;
    s.beta = beta;
    s.res = beta;
    s.jlast = s.jdone;
    s.jdone = 0;
    s.jmax = jmax;
    s.start_ok = beta <= tol ? 1 : 0;
    s.done = s.start_ok;
}

// start of a cycle: beta from the partial squared norms, V_0 = w / beta; the
// last block keeps the state
__global__ void __launch_bounds__(kVT)
gm_start_kernel(GmState st, double tol, const double *__restrict__ norms, int nb, const double2 *__restrict__ w,
                int64_t n, int64_t rows, double2 *__restrict__ v0) {
    __shared__ double red[1];
    const double beta = sqrt(block_norm_value(norms, nb, red));
    if (blockIdx.x == nb) {
        gm_begin(st, beta, tol, st.m);   // (the host ends the cycle)
        return;
    }
    scale_rows(w, beta > 0.0 ? 1.0 / beta : 0.0, n, rows, v0);
}

// Column j of H before its last rotation: the two passes' coefficients with the
// rotations of the columns before applied.
template <int T>
__device__ __forceinline__ void gm_rotate_column(const GmState &st, int j, const double2 *h2) {
    __shared__ double2 s_col[kHs + 1], s_sn[kHs + 1];
    __shared__ double s_cs[kHs + 1];
    double2 *out = st.H + (int64_t)j * (st.m + 1);
    const bool small = j < kHs;
    double2 *col = small ? s_col : out;
    const double2 *sn = small ? s_sn : st.sn;
    const double *cs = small ? s_cs : st.cs;
    for (int k = threadIdx.x; k <= j; k += T) {
        col[k] = make_double2(st.h1[k].x + h2[k].x, st.h1[k].y + h2[k].y);
        if (small && k < j) {
            s_sn[k] = st.sn[k];
            s_cs[k] = st.cs[k];
        }
    }
    __syncthreads();
    if (threadIdx.x < 4) rotate_column(col, sn, cs, j, threadIdx.x);
    __syncthreads();
    if (small)
        for (int k = threadIdx.x; k <= j; k += T) out[k] = col[k];
}

// w -= V h (ncol columns, h the sums of dots_in, or hsum already summed), then
// the partial dot products with V (first pass) or, LAST, the partial squared
// norms.  The first pass stores h in h1; in the last one a further block applies
// the earlier rotations to the new column of H.
template <int T, bool LAST>
__global__ void __launch_bounds__(T)
gm_update_kernel(GmState st, const double2 *__restrict__ V, int ncol, const double2 *__restrict__ dots_in,
                 const double2 *__restrict__ hsum, int nb, double2 *w, int64_t n, int64_t rows,
                 double2 *__restrict__ dots_out, double *__restrict__ norms, const int *__restrict__ stop) {
    if (stop && *stop) return;
    __shared__ double red[T];
    __shared__ double2 hs[kHs];
    const double2 *h = hsum;
    if (!hsum) {
        block_sums<T>(dots_in, nb, ncol, hs);
        __syncthreads();
        h = hs;
        if (!LAST && blockIdx.x == 0 && threadIdx.x < ncol) st.h1[threadIdx.x] = hs[threadIdx.x];
    }
    if (LAST && blockIdx.x == nb) {
        gm_rotate_column<T>(st, ncol - 1, h);
        return;
    }
    const int64_t r0 = (int64_t)blockIdx.x * rows, r1 = min(n, r0 + rows);
    double nrm = 0;
    over_rows<T>(r0, r1, red,
        [&](int64_t i, int g) {
            const bool im = i & 1;
            double s = 0;
#pragma unroll 8
            for (int c = g; c < ncol; c += kGroups<T>) {
                s = mul_step(s, V[(int64_t)c * n + (i >> 1)], h[c], im);
            }
            return s;
        },
        [&](int64_t i, double s, double) {
            const double v = comps(w)[i] - s;
            comps(w)[i] = v;
            if (LAST) nrm = fma(v, v, nrm);
        });
    if (LAST) {
        block_norm<T>(nrm, red, norms);
    } else {
        __syncthreads();
        block_dots<T>(V, n, ncol, w, r0, r1, dots_out, nb);
    }
}

// The last rotation of Arnoldi step j, residual estimate and stop test (cs
// real, sn complex), by one block: a = col[j] of H, hn2 = |w|^2.  Warps share the
// square roots, whose FP64 operations no warp can overlap.  |g_j| is the
// residual before the step.
__device__ __forceinline__ void gm_givens(const GmState &st, int j, const double *__restrict__ norms, int nb) {
    __shared__ double red[1], s_na2, s_ia, s_rh;
    GmScalars &s = *st.s;
    double2 *col = st.H + (int64_t)j * (st.m + 1);
    const double2 a = col[j], gj = st.g[j];   // (and g_{j+1} = 0)
    if (threadIdx.x == 32) {
        s_na2 = fma(a.x, a.x, a.y * a.y);
        s_ia = rsqrt(s_na2);
    }
    const double hn2 = block_norm_value(norms, nb, red), na2 = s_na2, ia = s_ia;
    if (threadIdx.x == 32) s_rh = rsqrt(hn2);
    double in = 0;
    if (threadIdx.x == 0) in = rsqrt(na2 + hn2);
    __syncthreads();
    if (threadIdx.x > 0) return;
    const Rotation rot = last_rotation(a, na2, ia, hn2, s_rh, in);
    const double res = s.res * rot.q;
    s.res = res;
    s.jdone = j + 1;
    if (res <= s.tol || hn2 == 0.0 || j + 1 >= s.jmax) s.done = 1;
    st.cs[j] = rot.c;
    st.sn[j] = rot.sn;
    col[j] = rot.r;
    col[j + 1] = make_double2(0.0, 0.0);
    const double2 ug = cmul(cconj(rot.sn), gj);
    st.g[j] = make_double2(rot.c * gj.x, rot.c * gj.y);
    st.g[j + 1] = make_double2(-ug.x, -ug.y);
}

// V_{j+1} = w / |w|, and in a further block the state of step j.  (A block that
// already sees the flag which that block raises skips a vector nothing reads.)
__global__ void __launch_bounds__(kVT)
gm_finish_kernel(GmState st, int j, const double *__restrict__ norms, int nb, const double2 *__restrict__ w, int64_t n,
                 int64_t rows, double2 *__restrict__ vn) {
    __shared__ double red[1];
    if (__syncthreads_or(threadIdx.x == 0 && *static_cast<volatile int *>(&st.s->done))) return;
    if (blockIdx.x == nb) {
        gm_givens(st, j, norms, nb);
        return;
    }
    const double hn2 = block_norm_value(norms, nb, red);
    scale_rows(w, hn2 > 0.0 ? rsqrt(hn2) : 0.0, n, rows, vn);
}

// y = R^{-1} g over the jdone columns (back substitution by columns, one warp)
__global__ void __launch_bounds__(32) gm_trisolve_kernel(GmState st) {
    constexpr int kS = 32;
    __shared__ double2 s_y[kS], s_R[kS * kS];
    const int j = st.s->jdone, ld = st.m + 1, lane = threadIdx.x;
    const bool small = j <= kS;
    double2 *y = small ? s_y : st.y;
    const double2 *R = small ? s_R : st.H;
    const int ldr = small ? kS : ld;
    for (int k = lane; k < j; k += 32) y[k] = st.g[k];
    if (small && lane < j)
#pragma unroll 8
        for (int k = 0; k < j; ++k) s_R[k * kS + lane] = st.H[(int64_t)k * ld + lane];
    __syncwarp();
    back_substitute(R, ldr, j, y, lane);
    if (small)
        for (int k = lane; k < j; k += 32) st.y[k] = y[k];
}

// x += V[:, 0..*ncol) yc  (column count on the device)
__global__ void combo_add_dev_kernel(const double2 *__restrict__ V, int64_t ldv, const int *__restrict__ ncol,
                                     const double2 *__restrict__ yc, double2 *__restrict__ x, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int nc = *ncol;
    double re = x[i].x, im = x[i].y;
#pragma unroll 4
    for (int c = 0; c < nc; ++c) {
        const double2 v = V[(int64_t)c * ldv + i], y = yc[c];
        re += v.x * y.x - v.y * y.y;
        im += v.x * y.y + v.y * y.x;
    }
    x[i] = make_double2(re, im);
}

// ---- graph form: the whole (refined) solve as conditional graph nodes --------
// Control flow lives in device memory (RfState) and in conditional handles that
// single-thread kernels set; every loop has a counter bound, so each WHILE node
// ends even for NaN residuals.
struct RfState {
    double bnorm, tol;     // |b| and the absolute tolerance max(reltol |b|, abstol)
    double res;            // last outer residual |b - A x| (exact product)
    double inner_tol;      // absolute tolerance of the current inner solve
    double last_beta;      // residual norm at the start of the last cycle
    long long matvecs;
    int iters, restarts, refinements;
    int outer_zero;        // x == 0: the outer residual is b (its product skipped)
    int inner_zero;        // dx == 0: the cycle residual is the right-hand side
    int steps, cycles;     // loop counters (bounds of the WHILE nodes)
    int pad;
};

// x += d
__global__ void axpy1_kernel(const double2 *__restrict__ d, double2 *__restrict__ x, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = make_double2(x[i].x + d[i].x, x[i].y + d[i].y);
}

// |b| from the norm reduction, tolerance, counters; enter the outer loop
__global__ void __launch_bounds__(32)
rf_start_kernel(RfState *rf, const double *__restrict__ norms, int nb, double reltol, double abstol,
                cudaGraphConditionalHandle h_outer) {
    __shared__ double red[1];
    const double bn = sqrt(block_norm_value(norms, nb, red));
    if (threadIdx.x > 0) return;
    RfState &r = *rf;
    r = RfState{};
    r.bnorm = bn;
    r.tol = fmax(reltol * bn, abstol);
    r.res = bn;
    r.last_beta = bn;
    r.outer_zero = 1;
    cudaGraphSetConditional(h_outer, 1u);
}

// Top of an outer pass.  Refinement: the outer residual |b - A x| decides
// whether another inner solve runs (the host loop of run_gmres); plain GMRES:
// one pass whose inner solve is the whole solve.
__global__ void __launch_bounds__(32)
rf_check_kernel(RfState *rf, const double *__restrict__ norms, int nb, int refine, int maxiter, int max_outer,
                double inner_rel, cudaGraphConditionalHandle h_outer, cudaGraphConditionalHandle h_cycle) {
    __shared__ double red[1];
    const double res = refine ? sqrt(block_norm_value(norms, nb, red)) : 0.0;
    if (threadIdx.x > 0) return;
    RfState &r = *rf;
    if (refine) {
        if (!r.outer_zero) r.matvecs += 1;
        r.outer_zero = 0;
        r.res = res;
        if (res <= r.tol || r.iters >= maxiter || r.refinements >= max_outer) {
            cudaGraphSetConditional(h_outer, 0u);
            cudaGraphSetConditional(h_cycle, 0u);
            return;
        }
        r.refinements += 1;
        r.inner_tol = fmax(inner_rel * res, r.tol * 0.5);
    } else {
        r.inner_tol = r.tol;
        cudaGraphSetConditional(h_outer, 0u);
    }
    r.inner_zero = 1;
    r.cycles = 0;
    cudaGraphSetConditional(h_cycle, 1u);
}

// Start of a restart cycle (gm_start_kernel with the inner tolerance read from
// the device); opens the Arnoldi loop unless the true residual already meets it.
__global__ void __launch_bounds__(kVT)
gm_cycle_start_kernel(GmState st, RfState *rf, int maxiter, int restart, const double *__restrict__ norms, int nb,
                      const double2 *__restrict__ w, int64_t n, int64_t rows, double2 *__restrict__ v0,
                      cudaGraphConditionalHandle h_step, cudaGraphConditionalHandle h_sel) {
    __shared__ double red[1];
    const double beta = sqrt(block_norm_value(norms, nb, red));
    if (blockIdx.x == nb) {
        RfState &r = *rf;
        const int jmax = min(restart, max(0, maxiter - r.iters));
        gm_begin(st, beta, r.inner_tol, jmax);
        if (threadIdx.x > 0) return;
        if (!r.inner_zero) r.matvecs += 1;
        r.inner_zero = 0;
        r.last_beta = beta;
        r.steps = 0;
        cudaGraphSetConditional(h_step, (!st.s->start_ok && jmax > 0) ? 1u : 0u);
        cudaGraphSetConditional(h_sel, 0u);
        return;
    }
    scale_rows(w, beta > 0.0 ? 1.0 / beta : 0.0, n, rows, v0);
}

// After each group of Arnoldi steps: the next group, and whether it runs (not
// converged, steps left in the cycle; at most `groups` passes)
__global__ void gm_step_guard_kernel(GmState st, RfState *rf, int groups, cudaGraphConditionalHandle h_step,
                                     cudaGraphConditionalHandle h_sel) {
    const GmScalars &s = *st.s;
    RfState &r = *rf;
    r.steps += 1;
    cudaGraphSetConditional(h_step, (!s.done && r.steps < groups) ? 1u : 0u);
    cudaGraphSetConditional(h_sel, (unsigned)r.steps);
}

// End of a cycle: tallies; another cycle (whose first action re-checks the true
// residual) follows any cycle that took steps
__global__ void gm_cycle_end_kernel(GmState st, RfState *rf, int maxiter, cudaGraphConditionalHandle h_cycle) {
    RfState &r = *rf;
    const int jd = st.s->jdone;
    r.iters += jd;
    r.matvecs += jd;
    if (jd > 0) r.restarts += 1;
    r.cycles += 1;
    cudaGraphSetConditional(h_cycle, (jd > 0 && r.cycles <= maxiter) ? 1u : 0u);
}

__global__ void rf_final_kernel(const RfState *rf, int refine, bie_gmres_info *out) {
    const RfState &r = *rf;
    bie_gmres_info o{};
    o.iterations = r.iters;
    o.restarts = r.restarts;
    o.refinements = refine ? r.refinements : 0;
    o.matvecs = r.matvecs;
    o.residual_norm = refine ? r.res : r.last_beta;
    o.rhs_norm = r.bnorm;
    o.converged = o.residual_norm <= r.tol ? 1 : 0;
    *out = o;
}

__global__ void round_c64_kernel(const double2 *__restrict__ in, float2 *__restrict__ out, int64_t n) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        out[i] = make_float2((float)in[i].x, (float)in[i].y);
}

inline unsigned blocks(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// Column slices of a dense product: as many as make one resident wave of
// blocks (the kernel's occupancy x the SMs) over the row tiles, so that no
// partial second wave trails the product (7842-node complex64 matrix: 5.1 ->
// 6.1 TB/s against a fixed 8 blocks per SM).
constexpr int kMaxSlices = 64;
inline int gemv_slices(const void *kern, int64_t rows, int num_sms) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kT, 0) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    const int64_t tiles = (rows + kT - 1) / kT;
    return (int)std::max<int64_t>(1, std::min<int64_t>(kMaxSlices, (int64_t)per_sm * num_sms / tiles));
}

// ---------------------------------------------------------------------------
// Operator application and BLAS-1 helpers bound to a context
// ---------------------------------------------------------------------------
struct Solver {
    Ctx &c;
    int64_t n;
    int m;                        // restart length
    RowSplit rs;                  // rows of the vector kernels' blocks
    double2 *part = nullptr;      // gemv slices
    double2 *dot1 = nullptr, *dot2 = nullptr;
    double *norms = nullptr;      // partial sums of the vector kernels
    GmState st{};                 // device-resident Arnoldi state
    RfState *rf = nullptr;        // device-resident refinement state (graph form)
    const void *slices_of = nullptr;   // kernel whose slices were asked for last
    int n_slices = 1;
    const int *stop = nullptr;    // device stop flag honoured by the launches below
    cudaStream_t stream;          // launch stream (a capture stream while recording a graph)
    DevOp *devop = nullptr;       // operator applied through DevOp::apply (else bie_operator)

    // level > 0: the workspace of a solve nested inside another solve's product
    Solver(Ctx &ctx, int64_t n_, int restart, int level = 0)
        : c(ctx), n(n_), m(restart), stream(ctx.stream) {
        const int part_slot = level == 0 ? kScratchSolverPart : kScratchSolverNested + 2 * (level - 1) + 1;
        rs = row_split(n);
        const size_t part_bytes = (size_t)kMaxSlices * n * 16;
        const size_t dot_bytes = (size_t)(restart + 1) * rs.nb * 16;
        const size_t nc = (size_t)(restart + 1) * restart + 4 * (size_t)(restart + 1) + restart;
        const size_t st_bytes = nc * 16 + (size_t)restart * 8 + sizeof(GmScalars) + sizeof(RfState) + 96;
        char *base = static_cast<char *>(
            c.scratch(part_slot, part_bytes + 2 * dot_bytes + (size_t)rs.nb * 16 + st_bytes));
        part = reinterpret_cast<double2 *>(base);
        dot1 = reinterpret_cast<double2 *>(base + part_bytes);
        dot2 = dot1 + (size_t)(restart + 1) * rs.nb;
        double2 *z = dot2 + (size_t)(restart + 1) * rs.nb;
        norms = reinterpret_cast<double *>(z);
        z += rs.nb;
        st.m = restart;
        st.H = z;
        z += (size_t)(restart + 1) * restart;
        st.g = z;
        z += restart + 1;
        st.sn = z;
        z += restart;
        st.h1 = z;
        z += restart + 1;
        st.h2 = z;
        z += restart + 1;
        st.y = z;
        z += restart + 1;
        st.cs = reinterpret_cast<double *>(z);
        st.s = reinterpret_cast<GmScalars *>(reinterpret_cast<char *>(st.cs) + (((size_t)restart * 8 + 15) & ~size_t(15)));
        rf = reinterpret_cast<RfState *>(reinterpret_cast<char *>(st.s) + ((sizeof(GmScalars) + 15) & ~size_t(15)));
    }

    void launched() { ++c.kernel_launches; }

    // y = s (K x) + d .* x up to the sum of its slices, which gm_product_kernel
    // takes (dense kernels skip when *stop is set)
    // slices of a product kernel over `rows` row threads (asked once per solver)
    int slices(const void *kern, int64_t rows) {
        if (kern != slices_of) {
            slices_of = kern;
            n_slices = gemv_slices(kern, rows, c.num_sms);
        }
        return n_slices;
    }
    Sliced product(const bie_operator &op, int precision, const double2 *x, double2 *y) {
        if (devop) {
            devop->apply(x, y, stop);
            return Sliced{};
        }
        const double2 sc = make_double2(op.scale_re, op.scale_im);
        const double2 *d = reinterpret_cast<const double2 *>(op.diag);
        if (op.kind == BIE_OP_DENSE) {
            cudaEvent_t t0 = c.timer_begin();
            int S = 1;
            if (op.A32 && (precision == BIE_PREC_MIXED || !op.A)) {
                // complex64 operator: the fast product for mixed iterations, the
                // exact one where FP64 arithmetic was asked for (residuals of
                // refinement, right-hand sides) and no complex128 matrix exists
                const bool exact = precision != BIE_PREC_MIXED;
                if (n % 2 == 0) {
                    if (exact) {
                        S = slices((const void *)dense_gemv_c64_exact_kernel, n / 2);
                        dense_gemv_c64_exact_kernel<<<dim3(blocks(n / 2, kT), (unsigned)S), kT, 0, stream>>>(
                            reinterpret_cast<const float4 *>(op.A32), n, x, part, S, stop);
                    } else {
                        S = slices((const void *)dense_gemv_c64_kernel, n / 2);
                        dense_gemv_c64_kernel<<<dim3(blocks(n / 2, kT), (unsigned)S), kT, 0, stream>>>(
                            reinterpret_cast<const float4 *>(op.A32), n, x, part, S, stop);
                    }
                } else {
                    if (exact) {
                        S = slices((const void *)dense_gemv_c64_rows_exact_kernel, n);
                        dense_gemv_c64_rows_exact_kernel<<<dim3(blocks(n, kT), (unsigned)S), kT, 0, stream>>>(
                            reinterpret_cast<const float2 *>(op.A32), n, x, part, S, stop);
                    } else {
                        S = slices((const void *)dense_gemv_c64_rows_kernel, n);
                        dense_gemv_c64_rows_kernel<<<dim3(blocks(n, kT), (unsigned)S), kT, 0, stream>>>(
                            reinterpret_cast<const float2 *>(op.A32), n, x, part, S, stop);
                    }
                }
            } else {
                S = slices((const void *)dense_gemv_kernel, n);
                dense_gemv_kernel<<<dim3(blocks(n, kT), (unsigned)S), kT, 0, stream>>>(
                    reinterpret_cast<const double2 *>(op.A), n, x, part, S, stop);
            }
            BIE_CUDA(cudaGetLastError());
            c.timer_end(t0);
            launched();
            return Sliced{part, S, sc, d, x};
        } else {
            // matrix-free F x (or the fast operator) into y, then y = s y + d .* x
            // (these products do not look at the stop flag: the caller checks it
            // on the host after every step)
            if (op.kind == BIE_OP_FAST) {
                FastOp &f = *const_cast<FastOp *>(reinterpret_cast<const FastOp *>(op.fast));
                apply_fastop(f, reinterpret_cast<const double *>(x), reinterpret_cast<double *>(y), precision,
                             nullptr, 0);
            } else {
                MatvecArgs mv{op.k_re, op.k_im, c.d_sources, n, reinterpret_cast<const double *>(x),
                              nullptr, reinterpret_cast<double *>(y), nullptr, precision};
                launch_matvec(c, mv);
            }
            return Sliced{y, 1, sc, d, x};
        }
    }

    // blocks of few rows or of many (over_rows)
    bool few() const { return rs.rows < kLongRows; }
    void finish_product(const Sliced &p, double2 *y, const double2 *rhs, const int *zero, const double2 *V, int ncol) {
        auto kern = few() ? gm_product_kernel<kVT> : gm_product_kernel<kVTLong>;
        kern<<<rs.nb, few() ? kVT : kVTLong, 0, stream>>>(p, n, rs.rows, y, rhs, zero, V, ncol, dot1, norms, stop);
        BIE_CUDA(cudaGetLastError());
        launched();
    }
    // y = s (K x) + d .* x
    void apply(const bie_operator &op, int precision, const double2 *x, double2 *y) {
        const Sliced p = product(op, precision, x, y);
        if (p.S > 0) finish_product(p, y, nullptr, nullptr, nullptr, 0);
    }
    // w = rhs - A x (rhs where *zero, whose product is skipped), partial norms
    void residual(const bie_operator &op, int precision, const double2 *rhs, const double2 *x, double2 *w,
                  const int *zero) {
        stop = zero;
        const Sliced p = product(op, precision, x, w);
        stop = nullptr;
        finish_product(p, w, rhs, zero, nullptr, -1);
    }

    // Arnoldi step j: w = A V_j, orthogonalised against V_0 .. V_j (CGS2), V_{j+1}
    void arnoldi_step(const bie_operator &op, int precision, double2 *V, double2 *w, int j) {
        const int nc = j + 1;
        const Sliced p = product(op, precision, V + (int64_t)j * n, w);
        finish_product(p, w, nullptr, nullptr, V, nc);
        for (int pass = 0; pass < 2; ++pass) {
            const double2 *in = pass ? dot2 : dot1;
            const double2 *hsum = nullptr;
            if (nc > kHs) {
                double2 *h = pass ? st.h2 : st.h1;
                sum_partials_kernel<<<blocks(nc, kT / 32), kT, 0, stream>>>(in, rs.nb, nc, h, stop);
                BIE_CUDA(cudaGetLastError());
                launched();
                hsum = h;
            }
            auto kern = pass ? (few() ? gm_update_kernel<kVT, true> : gm_update_kernel<kVTLong, true>)
                             : (few() ? gm_update_kernel<kVT, false> : gm_update_kernel<kVTLong, false>);
            kern<<<rs.nb + pass, few() ? kVT : kVTLong, 0, stream>>>(st, V, nc, in, hsum, rs.nb, w, n, rs.rows, dot2,
                                                                    norms, stop);
            BIE_CUDA(cudaGetLastError());
            launched();
        }
        gm_finish_kernel<<<rs.nb + 1, kVT, 0, stream>>>(st, j, norms, rs.nb, w, n, rs.rows, V + (int64_t)nc * n);
        BIE_CUDA(cudaGetLastError());
        launched();
    }

    // x += V y, R y = g
    void add_solution(const double2 *V, double2 *x) {
        gm_trisolve_kernel<<<1, 32, 0, stream>>>(st);
        BIE_CUDA(cudaGetLastError());
        launched();
        combo_add_dev_kernel<<<blocks(n, 64), 64, 0, stream>>>(V, n, &st.s->jdone, st.y, x, n);
        BIE_CUDA(cudaGetLastError());
        launched();
    }

    // partial squared norms of w
    void norm_partials(const double2 *w) {
        finish_product(Sliced{}, const_cast<double2 *>(w), nullptr, nullptr, nullptr, -1);
    }
    // the norm from these
    double norm_value() {
        std::vector<double> h(rs.nb);
        BIE_CUDA(cudaMemcpyAsync(h.data(), norms, h.size() * sizeof(double), cudaMemcpyDeviceToHost, stream));
        BIE_CUDA(cudaStreamSynchronize(stream));
        double s = 0;
        for (double v : h) s += v;
        return std::sqrt(std::max(s, 0.0));
    }
};

// One GMRES solve of A x = b from the initial x (device), operator precision
// `prec`; returns the number of iterations; `tol` is an absolute tolerance on
// the residual norm.  V: (restart + 1) x n workspace.
//
// Each restart cycle runs on the device without host round trips: the
// Gram-Schmidt coefficients, the Hessenberg column, the Givens rotations and
// the residual estimate stay in device memory (GmState), one block of a step
// decides convergence and raises a stop flag, and every later kernel of
// the cycle returns at once when it sees the flag.  The host reads the state
// once per cycle (dense operators) or once per step (matrix-free and fast
// operators, whose products do not look at the flag).
int gmres_core(Solver &S, const bie_operator &op, int prec, const double2 *b, double2 *x,
               bool x_zero, double2 *V, double2 *w, int restart, int maxiter, double tol,
               double *res_out, int *restarts_out, int64_t *matvecs) {
    const int64_t n = S.n;
    const bool dense = S.devop ? S.devop->honours_stop() : op.kind == BIE_OP_DENSE;
    const GmState st = S.st;
    const int *stop_flag = &st.s->done;
    cudaStream_t stream = S.stream;
    int it = 0, restarts = 0;
    double beta = 0.0;
    GmScalars hs{};
    for (bool first = true;; first = false) {
        // r = b - A x  (r = b for a zero start), beta = |r|
        if (first && x_zero) {
            BIE_CUDA(cudaMemcpyAsync(w, b, (size_t)n * 16, cudaMemcpyDeviceToDevice, stream));
            S.stop = nullptr;
            S.norm_partials(w);
        } else {
            S.residual(op, prec, b, x, w, nullptr);
            ++*matvecs;
        }
        gm_start_kernel<<<S.rs.nb + 1, kVT, 0, stream>>>(st, tol, S.norms, S.rs.nb, w, n, S.rs.rows, V);
        BIE_CUDA(cudaGetLastError());
        S.launched();
        BIE_CUDA(cudaMemcpyAsync(&hs, st.s, sizeof(GmScalars), cudaMemcpyDeviceToHost, stream));
        BIE_CUDA(cudaStreamSynchronize(stream));
        if (!first) {
            it += hs.jlast;
            *matvecs += hs.jlast;
            ++restarts;
        }
        const int jmax = std::min(restart, std::max(0, maxiter - it));
        if (hs.start_ok || jmax == 0) {
            beta = hs.beta;
            break;
        }
        S.stop = stop_flag;
        for (int j = 0; j < jmax; ++j) {
            S.arnoldi_step(op, prec, V, w, j);
            // the host looks at the stop flag after every step for operators whose
            // products ignore it, every kCheck steps for dense ones (at most
            // kCheck - 1 skipped steps are queued after convergence)
            constexpr int kCheck = 4;
            if (!dense || j % kCheck == kCheck - 1) {
                int done = 0;
                BIE_CUDA(cudaMemcpyAsync(&done, stop_flag, sizeof(int), cudaMemcpyDeviceToHost, stream));
                BIE_CUDA(cudaStreamSynchronize(stream));
                if (done) break;
            }
        }
        S.stop = nullptr;
        S.add_solution(V, x);
    }
    *res_out = beta;
    *restarts_out = restarts;
    return it;
}

}  // namespace

// A conditional handle of the graph being captured on `s`.
cudaGraphConditionalHandle graph_new_handle(cudaStream_t s) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaGraph_t g = nullptr;
    BIE_CUDA(cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, nullptr, nullptr, nullptr));
    if (cs != cudaStreamCaptureStatusActive) fail(BIE_ERR_INVALID, "graph GMRES: the stream is not capturing");
    cudaGraphConditionalHandle h;
    BIE_CUDA(cudaGraphConditionalHandleCreate(&h, g, 0, 0));
    return h;
}

// Appends a conditional node after the capture's current dependencies; its body
// graphs are returned for capture on other streams.
void graph_add_conditional(cudaStream_t s, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type,
                           unsigned size, cudaGraph_t *bodies) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t *deps = nullptr;
    size_t nd = 0;
    BIE_CUDA(cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, nullptr, &nd));
    if (cs != cudaStreamCaptureStatusActive) fail(BIE_ERR_INVALID, "graph GMRES: the stream is not capturing");
    cudaGraphNodeParams p{};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = type;
    p.conditional.size = size;
    cudaGraphNode_t node;
    BIE_CUDA(cudaGraphAddNode(&node, g, deps, nullptr, nd, &p));
    BIE_CUDA(cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    for (unsigned i = 0; i < size; ++i) bodies[i] = p.conditional.phGraph_out[i];
}

constexpr int kStepGroup = 4;   // Arnoldi steps per pass of the graph form's loop

void capture_gmres(Ctx &c, const bie_operator &op, const double *b_, double *x_, const bie_gmres_opts &o,
                   bie_gmres_info *d_info, const cudaStream_t *body) {
    if (op.kind != BIE_OP_DENSE) fail(BIE_ERR_UNSUPPORTED, "graph GMRES needs a dense operator");
    if (o.initially_nonzero) fail(BIE_ERR_UNSUPPORTED, "graph GMRES starts from x = 0");
    const int64_t n = c.n_sources;
    const int restart = (int)std::max<int64_t>(1, std::min<int64_t>(o.restart > 0 ? o.restart : 20, n));
    if (restart > kGraphMaxRestart) fail(BIE_ERR_UNSUPPORTED, "graph GMRES: restart above 64");
    const int maxiter = o.maxiter > 0 ? o.maxiter : (int)std::min<int64_t>(n, INT32_MAX);
    const double reltol = o.reltol > 0 ? o.reltol : std::sqrt(2.220446049250313e-16);
    const double abstol = std::max(0.0, o.abstol);
    const bool refine = o.refine != 0;
    const int prec = refine ? BIE_PREC_MIXED : o.precision;
    const double inner_rel = o.inner_reltol > 0 ? o.inner_reltol : 1e-4;
    const int max_outer = o.max_refine > 0 ? o.max_refine : 10;
    const double2 *b = reinterpret_cast<const double2 *>(b_);
    double2 *x = reinterpret_cast<double2 *>(x_);

    char *ws = static_cast<char *>(c.scratch(kScratchSolver, (size_t)(restart + 4) * n * 16));
    double2 *V = reinterpret_cast<double2 *>(ws);
    double2 *w = V + (int64_t)(restart + 1) * n;
    double2 *rr = w + n;
    double2 *dx = rr + n;
    Solver S(c, n, restart);
    const GmState st = S.st;
    RfState *rf = S.rf;
    cudaStream_t s0 = c.stream;

    BIE_CUDA(cudaMemsetAsync(x, 0, (size_t)n * 16, s0));
    S.norm_partials(b);
    const cudaGraphConditionalHandle h_outer = graph_new_handle(s0);
    rf_start_kernel<<<1, 32, 0, s0>>>(rf, S.norms, S.rs.nb, reltol, abstol, h_outer);
    BIE_CUDA(cudaGetLastError());
    S.launched();
    cudaGraph_t g_outer;
    graph_add_conditional(s0, h_outer, cudaGraphCondTypeWhile, 1, &g_outer);
    {
        // outer pass: refinement residual rr = b - A x (exact product), then the
        // inner restarted GMRES on A dx = rr
        BodyCapture bc1(body[0], g_outer);
        S.stream = body[0];
        if (refine) {
            S.residual(op, o.precision == BIE_PREC_DF64 ? BIE_PREC_DF64 : BIE_PREC_FP64, b, x, rr, &rf->outer_zero);
            BIE_CUDA(cudaMemsetAsync(dx, 0, (size_t)n * 16, S.stream));
        }
        const double2 *rhs = refine ? rr : b;
        double2 *sol = refine ? dx : x;
        const cudaGraphConditionalHandle h_cycle = graph_new_handle(S.stream);
        rf_check_kernel<<<1, 32, 0, S.stream>>>(rf, S.norms, S.rs.nb, refine ? 1 : 0, maxiter, max_outer, inner_rel,
                                                h_outer, h_cycle);
        BIE_CUDA(cudaGetLastError());
        S.launched();
        cudaGraph_t g_cycle;
        graph_add_conditional(S.stream, h_cycle, cudaGraphCondTypeWhile, 1, &g_cycle);
        {
            // restart cycle: w = rhs - A sol (rhs itself on the first cycle), beta,
            // then up to `restart` Arnoldi steps
            BodyCapture bc2(body[1], g_cycle);
            S.stream = body[1];
            S.residual(op, prec, rhs, sol, w, &rf->inner_zero);
            const cudaGraphConditionalHandle h_step = graph_new_handle(S.stream);
            const cudaGraphConditionalHandle h_sel = graph_new_handle(S.stream);
            gm_cycle_start_kernel<<<S.rs.nb + 1, kVT, 0, S.stream>>>(st, rf, maxiter, restart, S.norms, S.rs.nb, w, n,
                                                                   S.rs.rows, V, h_step, h_sel);
            BIE_CUDA(cudaGetLastError());
            S.launched();
            cudaGraph_t g_step;
            graph_add_conditional(S.stream, h_step, cudaGraphCondTypeWhile, 1, &g_step);
            {
                // kStepGroup Arnoldi steps per pass: a switch over the group runs the
                // body recorded for its steps (CGS2 over j + 1 basis vectors for step
                // j); steps after the last one skip.  Solves of 8 wavenumbers at 2562
                // nodes: 7.9 ms with 1 step per pass, 7.8 with 2, 7.6 with 4, 7.7 with 8.
                BodyCapture bc3(body[2], g_step);
                S.stream = body[2];
                const int groups = (restart + kStepGroup - 1) / kStepGroup;
                std::vector<cudaGraph_t> branch(groups);
                graph_add_conditional(S.stream, h_sel, cudaGraphCondTypeSwitch, (unsigned)groups, branch.data());
                gm_step_guard_kernel<<<1, 1, 0, S.stream>>>(st, rf, groups, h_step, h_sel);
                BIE_CUDA(cudaGetLastError());
                S.launched();
                S.stop = &st.s->done;
                for (int g = 0; g < groups; ++g) {
                    BodyCapture bc4(body[3], branch[g]);
                    S.stream = body[3];
                    for (int j = g * kStepGroup; j < std::min(restart, (g + 1) * kStepGroup); ++j)
                        S.arnoldi_step(op, prec, V, w, j);
                    bc4.end();
                }
                S.stop = nullptr;
                bc3.end();
            }
            S.stream = body[1];
            S.add_solution(V, sol);
            gm_cycle_end_kernel<<<1, 1, 0, S.stream>>>(st, rf, maxiter, h_cycle);
            BIE_CUDA(cudaGetLastError());
            S.launched();
            bc2.end();
        }
        S.stream = body[0];
        if (refine) {
            axpy1_kernel<<<blocks(n), 256, 0, S.stream>>>(dx, x, n);
            BIE_CUDA(cudaGetLastError());
            S.launched();
        }
        bc1.end();
    }
    S.stream = s0;
    rf_final_kernel<<<1, 1, 0, s0>>>(rf, refine ? 1 : 0, d_info);
    BIE_CUDA(cudaGetLastError());
    S.launched();
}

namespace {

// The restarted (optionally refined) GMRES behind run_gmres and run_gmres_devop.
void gmres_solve(Ctx &c, const bie_operator &op, DevOp *devop, int64_t n, int level, const double *b_,
                 double *x_, const bie_gmres_opts &o, bie_gmres_info &info) {
    if (level < 0 || level > kMaxSolveLevel) fail(BIE_ERR_INVALID, "GMRES nesting deeper than two levels");
    const int restart = (int)std::max<int64_t>(1, std::min<int64_t>(o.restart > 0 ? o.restart : 20, n));
    const int maxiter = o.maxiter > 0 ? o.maxiter : (int)std::min<int64_t>(n, INT32_MAX);
    const double reltol = o.reltol > 0 ? o.reltol : std::sqrt(2.220446049250313e-16);
    const double abstol = std::max(0.0, o.abstol);
    const double2 *b = reinterpret_cast<const double2 *>(b_);
    double2 *x = reinterpret_cast<double2 *>(x_);

    // workspace: V (restart + 1) x n, w, r, dx
    const int ws_slot = level == 0 ? kScratchSolver : kScratchSolverNested + 2 * (level - 1);
    char *ws = static_cast<char *>(c.scratch(ws_slot, (size_t)(restart + 4) * n * 16));
    double2 *V = reinterpret_cast<double2 *>(ws);
    double2 *w = V + (int64_t)(restart + 1) * n;
    double2 *rr = w + n;
    double2 *dx = rr + n;
    Solver S(c, n, restart, level);
    S.devop = devop;
    S.norm_partials(b);
    const double bnorm = S.norm_value();
    const double tol = std::max(reltol * bnorm, abstol);
    if (!o.initially_nonzero) BIE_CUDA(cudaMemsetAsync(x, 0, (size_t)n * 16, c.stream));
    int64_t matvecs = 0;
    int iters = 0, restarts = 0;
    double res = 0;
    int outer = 0;
    if (!o.refine) {
        const int prec = o.precision;
        iters = gmres_core(S, op, prec, b, x, !o.initially_nonzero, V, w, restart, maxiter, tol, &res,
                           &restarts, &matvecs);
    } else {
        // iterative refinement: r = b - A x in FP64; inner solve A_low dx = r
        const double inner_rel = o.inner_reltol > 0 ? o.inner_reltol : 1e-4;
        const int max_outer = o.max_refine > 0 ? o.max_refine : 10;
        bie_operator low = op;
        for (outer = 0; outer < max_outer; ++outer) {
            S.residual(op, o.precision == BIE_PREC_DF64 ? BIE_PREC_DF64 : BIE_PREC_FP64, b, x, rr, nullptr);
            ++matvecs;
            res = S.norm_value();
            if (res <= tol || iters >= maxiter) break;
            BIE_CUDA(cudaMemsetAsync(dx, 0, (size_t)n * 16, c.stream));
            double ires = 0;
            int irs = 0;
            iters += gmres_core(S, low, BIE_PREC_MIXED, rr, dx, true, V, w, restart, maxiter - iters,
                                std::max(inner_rel * res, tol * 0.5), &ires, &irs, &matvecs);
            restarts += irs;
            axpy1_kernel<<<blocks(n), 256, 0, c.stream>>>(dx, x, n);
            BIE_CUDA(cudaGetLastError());
            S.launched();
        }
    }
    BIE_CUDA(cudaStreamSynchronize(c.stream));
    info.iterations = iters;
    info.restarts = restarts;
    info.refinements = outer;
    info.matvecs = matvecs;
    info.residual_norm = res;
    info.rhs_norm = bnorm;
    info.converged = res <= tol ? 1 : 0;
}

}  // namespace

void run_gmres(Ctx &c, const bie_operator &op, const double *b, double *x, const bie_gmres_opts &o,
               bie_gmres_info &info) {
    gmres_solve(c, op, nullptr, c.n_sources, 0, b, x, o, info);
}

void run_gmres_devop(Ctx &c, DevOp &op, const double *b, double *x, const bie_gmres_opts &o,
                     bie_gmres_info &info, int level) {
    bie_gmres_opts plain = o;
    plain.refine = 0;   // one arithmetic: the operator's own
    bie_operator none{};
    none.kind = -1;
    gmres_solve(c, none, &op, op.size(), level, b, x, plain, info);
}

void apply_operator(Ctx &c, const bie_operator &op, int precision, const double *x, double *y) {
    Solver S(c, c.n_sources, 1);
    S.apply(op, precision, reinterpret_cast<const double2 *>(x), reinterpret_cast<double2 *>(y));
}

void round_to_c64(Ctx &c, const double *in, float *out, int64_t n) {
    round_c64_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 64LL * c.num_sms), 256, 0, c.stream>>>(
        reinterpret_cast<const double2 *>(in), reinterpret_cast<float2 *>(out), n);
    BIE_CUDA(cudaGetLastError());
    ++c.kernel_launches;
}

}  // namespace bie
