// Exact propagators of linear absorption, built and applied: Propagation Diagonal,
// and Propagation Sparse where the static-coupling Taylor route does not
// apply (HamiltonianType Full, or a Threshold that truncates U).
//
// The reference computes, per vector and per step, the full one-step
// propagator U = V diag(exp(-i e f)) V^T from an FP32 LAPACK ssyev of the
// frame and applies it (propagate_vec_DIA, propagate.c:60-125), or applies
// only the elements with |U_ab|^2 > Threshold (propagate_vec_DIA_S,
// :185-258; Threshold pre-scaled by (f/ts)^2 at input, readinput.c:264-267).
// Here U is built once per frame in FP64 (propagators.cu; with kernel_config 2
// from an eigendecomposition, eigen.cu and k_build_u), rounded to the working
// precision, truncated by the same test in the working precision, and shared
// by every start point and polarisation that crosses the frame.  U is complex
// symmetric, so it is stored once and read along rows.
#include <algorithm>

#include "common.cuh"
#include "engine.h"

namespace {

// U[t][a][c] for the frames of one eigen chunk: CTA per frame, V^T and the
// phases in shared memory, one packed (a <= c) element per thread-iteration,
// mirrored so that U is exactly symmetric.
template <typename R>
__global__ void k_build_u(const double *V, const double *w, int n, double f, float thres, int truncate,
                          typename Vec2<R>::T *U) {
    typedef typename Vec2<R>::T R2;
    extern __shared__ double sh[];
    double *Vt = sh, *ph = Vt + (size_t)n * n;  // Vt[k][a] = V[a][k]; ph[2k], ph[2k+1]
    const double *Vf = V + (size_t)blockIdx.x * n * n;
    const double *wf = w + (size_t)blockIdx.x * n;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        int a = e / n, k = e % n;
        Vt[(size_t)k * n + a] = Vf[e];
    }
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        double s, c;
        sincos(wf[k] * f, &s, &c);
        ph[2 * k] = c;
        ph[2 * k + 1] = -s;
    }
    __syncthreads();
    R2 *Uf = U + (size_t)blockIdx.x * n * n;
    const int np = n * (n + 1) / 2;
    for (int e = threadIdx.x; e < np; e += blockDim.x) {
        // packed upper-triangle e -> (a, c), a <= c
        int a = 0, rem = e;
        while (rem >= n - a) { rem -= n - a; a++; }
        int c = a + rem;
        double ur = 0, ui = 0;
        for (int k = 0; k < n; k++) {
            double p = Vt[(size_t)k * n + a] * Vt[(size_t)k * n + c];
            ur = fma(p, ph[2 * k], ur);
            ui = fma(p, ph[2 * k + 1], ui);
        }
        R2 z;
        z.x = (R)ur;
        z.y = (R)ui;
        if (truncate) {
            bool keep;
            if (sizeof(R) == 4)
                keep = __fadd_rn(__fmul_rn((float)z.x, (float)z.x), __fmul_rn((float)z.y, (float)z.y)) > thres;
            else
                keep = (double)z.x * z.x + (double)z.y * z.y > (double)thres;
            if (!keep) z.x = z.y = (R)0;
        }
        Uf[(size_t)a * n + c] = z;
        Uf[(size_t)c * n + a] = z;
    }
}

// Linear absorption with per-frame propagators: CTA per start point, its
// three polarisation vectors in shared memory.  The response is taken before
// each step (absorption.c:119-145): float products, double sums.  The step is
// c_a <- sum_b U_ab c_b in site order b, the reference's float accumulation
// (propagate.c:109-119) in FP32 mode, so its parallelism is rows x vectors: a
// thread per row of VX vectors (one each while 3 n threads and three warps for
// the responses fit a CTA, else all three).  Where two U_t fit shared memory
// (STAGE) the next one is copied asynchronously while the sums run.  Bound by
// the chain of a row's additions and the issue of its few warps.  48 sites, 94
// start points, RunTimes 128: 1756 us with 64 threads that fetched U when
// needed, 175 us now (216 with the sums split over 19 groups of rows: the
// barriers of 1024 threads cost more than the shorter chains save, and another
// rounding).
template <typename R, int VX, bool STAGE>
__global__ void __launch_bounds__(1024) k_abs_dia(DevTraj T, const typename Vec2<R>::T *__restrict__ U, long f0, int n,
                                                  int rw, AbsJob J, double2 *resp) {
    typedef typename Vec2<R>::T R2;
    typedef Ar<R> A;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R2 *C = (R2 *)smem_raw, *D = C + 3 * n, *Us = D + 3 * n;  // [3][n] twice; [2][n][n] (STAGE)
    const int work = VX == 1 ? 3 * n : n, a = threadIdx.x % n, x0 = VX == 1 ? threadIdx.x / n : 0, lane = threadIdx.x & 31;
    const int x = (int)(threadIdx.x >> 5) - rw;  // the response warps: x = 0, 1, 2
    const bool act = (int)threadIdx.x < work;
    const size_t nn = (size_t)n * n;
    const int sl = blockIdx.x;
    const long ti = (long)(J.begin + sl) * J.sample;
    const R2 *Ut = U + (size_t)(ti - f0) * nn;
    for (int e = threadIdx.x; e < 3 * n; e += blockDim.x) {
        C[e].x = (R)traj_mu(T, ti, e / n, e % n);
        C[e].y = 0;
    }
    auto stage = [&](int t1) {
        if (t1 < J.tmax - 1)
            for (int e = threadIdx.x; e < (int)nn; e += blockDim.x)
                asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(Us + (t1 & 1) * nn + e)),
                             "l"(Ut + (size_t)t1 * nn + e), "n"(sizeof(R2)));
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (STAGE) stage(0);
    for (int t1 = 0; t1 < J.tmax; t1++) {
        if (STAGE) asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // U_t1 staged, C complete
        if (STAGE) stage(t1 + 1);
        if (x >= 0 && x < 3) {
            const long t = ti + t1;
            double re = 0, im = 0;
            for (int i = lane; i < n; i += 32) {
                const R m = (R)traj_mu(T, t, x, i);
                re += (double)A::mul(m, C[x * n + i].x);
                im += (double)A::mul(m, C[x * n + i].y);
            }
            for (int o = 16; o > 0; o >>= 1) {
                re += __shfl_xor_sync(0xffffffffu, re, o);
                im += __shfl_xor_sync(0xffffffffu, im, o);
            }
            if (lane == 0) resp[(size_t)(3 * sl + x) * J.tmax + t1] = make_double2(re, im);
        }
        if (t1 == J.tmax - 1) break;
        if (act) {
            const R2 *Ua = (STAGE ? Us + (t1 & 1) * nn : Ut + (size_t)t1 * nn) + a;
            R2 acc[VX];
#pragma unroll
            for (int q = 0; q < VX; q++) acc[q].x = acc[q].y = 0;
#pragma unroll 8
            for (int b = 0; b < n; b++) {
                const R2 u = Ua[(size_t)b * n];  // = U[a][b]
#pragma unroll
                for (int q = 0; q < VX; q++) {
                    const R2 z = C[(x0 + q) * n + b];
                    acc[q].x = A::add(acc[q].x, A::sub(A::mul(u.x, z.x), A::mul(u.y, z.y)));
                    acc[q].y = A::add(acc[q].y, A::add(A::mul(u.x, z.y), A::mul(u.y, z.x)));
                }
            }
#pragma unroll
            for (int q = 0; q < VX; q++) D[(x0 + q) * n + a] = acc[q];
        }
        R2 *sw = C;
        C = D;
        D = sw;
    }
}

}  // namespace

namespace {
template <typename R>
int run_abs_dia(const DevTraj &T, const typename Vec2<R>::T *U, long f0, int n, const AbsJob &J, double2 *resp,
                cudaStream_t s) {
    const bool one = 3 * n <= 928;  // a vector per thread
    const int work = ((one ? 3 * n : n) + 31) / 32 * 32;
    const bool own = work + 96 <= 1024;  // above 928 sites the first three warps take the responses too
    const int threads = own ? work + 96 : work;
    const size_t base = sizeof(typename Vec2<R>::T) * 6 * (size_t)n, all = base + sizeof(typename Vec2<R>::T) * 2 * n * n;
    const bool stage = one && all <= 227 * 1024;
    const size_t sm = stage ? all : base;
    auto kern = stage ? k_abs_dia<R, 1, true> : one ? k_abs_dia<R, 1, false> : k_abs_dia<R, 3, false>;
    if (const int e = allow_smem(kern, sm)) return e;
    kern<<<J.nsamp, threads, sm, s>>>(T, U, f0, n, own ? work / 32 : 0, J, resp);
    return (int)cudaGetLastError();
}
}  // namespace

size_t dia_build_smem(int n) { return sizeof(double) * ((size_t)n * n + 2 * n); }

int launch_build_u(int prec, const double *V, const double *w, long nfr, int n, double f, float thres, int truncate,
                   void *U, cudaStream_t s) {
    if (nfr <= 0) return 0;
    size_t sm = dia_build_smem(n);
    int e;
    if (prec == 0) {
        if ((e = allow_smem(k_build_u<float>, sm))) return e;
        k_build_u<float><<<(unsigned)nfr, 256, sm, s>>>(V, w, n, f, thres, truncate, (float2 *)U);
    } else {
        if ((e = allow_smem(k_build_u<double>, sm))) return e;
        k_build_u<double><<<(unsigned)nfr, 256, sm, s>>>(V, w, n, f, thres, truncate, (double2 *)U);
    }
    return (int)cudaGetLastError();
}

int launch_abs_dia(int prec, const DevTraj &T, const void *U, long f0, int n, const AbsJob &J, double2 *resp,
                   cudaStream_t s) {
    if (J.nsamp <= 0) return 0;
    if (n > 1024) return (int)cudaErrorNotSupported;
    return prec == 0 ? run_abs_dia<float>(T, (const float2 *)U, f0, n, J, resp, s)
                     : run_abs_dia<double>(T, (const double2 *)U, f0, n, J, resp, s);
}
