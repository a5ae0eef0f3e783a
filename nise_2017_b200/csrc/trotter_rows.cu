// Linear absorption with the Trotter scheme on rows of operations (rows.cuh): a
// warp per vector on rows of 32, two warps on rows of 64; the same responses as
// the other Trotter kernels.
#include "common.cuh"
#include "engine.h"
#include "rows.cuh"
#include "schemes.cuh"

namespace {

template <typename R, int TW>
__global__ void __launch_bounds__(256) k_abs_trotter_rows(DevTraj T, SinglesTab D, RowPlan Q, AbsJob J, double2 *resp,
                                                          int nvec, int stage) {
    typedef typename Vec2<R>::T R2;
    typedef Ar<R> A;
    constexpr int W = 32 * TW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const R2 *rs;
    R2 *X = rows_setup<R, TW>(D, Q, stage, smem_raw, rs);
    const int n = D.n, th = threadIdx.x % W, bar = 1 + threadIdx.x / W, v = blockIdx.x * (blockDim.x / W) + threadIdx.x / W;
    if (v >= nvec) return;
    const int x = v % 3;
    const long ti = (long)(J.begin + v / 3) * J.sample;
    for (int a = th; a < n; a += W) {
        R2 z;
        z.x = (R)traj_mu(T, ti, x, a);
        z.y = 0;
        X[a] = z;
    }
    for (int t1 = 0; t1 < J.tmax; t1++) {
        rows_sync<TW>(bar);
        if (th < 32) {  // the first warp takes the response (dot_mu's order)
            double re = 0, im = 0;
#pragma unroll 4
            for (int a = th; a < n; a += 32) {
                const R m = (R)traj_mu(T, ti + t1, x, a);
                re += (double)A::mul(m, X[a].x);
                im += (double)A::mul(m, X[a].y);
            }
            const double2 z = resp_sum_warp(re, im, n);
            if (th == 0) resp[(size_t)v * J.tmax + t1] = z;
        }
        if (t1 < J.tmax - 1) rows_singles_step<R, TW>(D, Q, X, rs, th, bar, ti + t1 - D.f0);
    }
}

template <typename R, int TW>
int run(const DevTraj &T, const SinglesTab &D, const RowPlan &Q, const AbsJob &J, double2 *resp, cudaStream_t s) {
    const int nvec = 3 * J.nsamp;
    const RowShape h = rows_shape<R>(D.n, D.K, D.rot_static, Q.nrow, TW, nvec, sm_count());
    if (!h.vecs) return (int)cudaErrorNotSupported;
    if (const int e = allow_smem(k_abs_trotter_rows<R, TW>, h.bytes)) return e;
    k_abs_trotter_rows<R, TW><<<(nvec + h.vecs - 1) / h.vecs, 32 * TW * h.vecs, h.bytes, s>>>(T, D, Q, J, resp, nvec,
                                                                                             h.stage);
    return (int)cudaGetLastError();
}

}  // namespace

bool trotter_rows_fit(int prec, const TrotterPlan &P, const RowPlan &Q, int width) {
    if (!Q.ab) return false;
    return (prec == 0 ? rows_shape<float>(P.n, P.k, P.rot_static, Q.nrow, width / 32, 1, 1)
                      : rows_shape<double>(P.n, P.k, P.rot_static, Q.nrow, width / 32, 1, 1))
               .vecs > 0;
}

int trotter_rows_vecs(int prec, const TrotterPlan &P, const RowPlan &Q, int width, int nvec) {
    if (!Q.ab) return 0;
    const RowShape h = prec == 0 ? rows_shape<float>(P.n, P.k, P.rot_static, Q.nrow, width / 32, nvec, sm_count())
                                 : rows_shape<double>(P.n, P.k, P.rot_static, Q.nrow, width / 32, nvec, sm_count());
    return h.stage ? h.vecs : 0;
}

int launch_abs_trotter_rows(int prec, const DevTraj &T, const TrotterPlan &P, const RowPlan &Q, int width,
                            const AbsJob &J, double2 *resp, cudaStream_t s) {
    if (J.nsamp <= 0) return 0;
    SinglesTab D = {};
    D.n = P.n;
    D.ts = J.ts;
    D.f0 = P.f0;
    D.K = P.k;
    D.U = P.U;
    D.rot = P.rot;
    D.rot_static = P.rot_static;
    if (width == 64) return prec == 0 ? run<float, 2>(T, D, Q, J, resp, s) : run<double, 2>(T, D, Q, J, resp, s);
    return prec == 0 ? run<float, 1>(T, D, Q, J, resp, s) : run<double, 1>(T, D, Q, J, resp, s);
}
