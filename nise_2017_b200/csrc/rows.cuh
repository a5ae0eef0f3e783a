// One Trotter time step of a vector on a warp (or two), from the rows of
// nise_row_schedule: the lanes apply the operations of a row (rotations and
// half-step phases alike, both 2x2 on two sites of the state in shared memory), a
// __syncwarp separates the rows.  Sub-steps overlap as far as the couplings
// allow, so a step has about (couplings + 2 sites) x sub-steps / 32 rows (64
// sites, all coupled, 5 sub-steps: 396; a 16-site chain: 33) instead of that many
// operations in sequence on a thread.  Every site sees the float operations of
// trotter_apply in their order, so the results are bitwise the same.  Bound by a
// row's latency: two loads of the state, a multiply and an add, the stores.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "rotsched.h"

// The coefficients of an entry, from the frame's rotations and phases.
template <typename R>
__device__ __forceinline__ typename Vec2<R>::T row_coef(unsigned y, const typename Vec2<R>::T *rot,
                                                        const typename Vec2<R>::T *ph) {
    return ((y & NISE_ROW_PHASE) ? ph : rot)[y & ~NISE_ROW_PHASE];
}

// The threads of a vector: one warp, or two on rows of 64 (a named barrier
// separates the rows then; id 1 and up, 0 is __syncthreads).
template <int TW> __device__ __forceinline__ void rows_sync(int bar) {
    if (TW == 1) __syncwarp();
    else asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
}

// X [n + 32 TW] state (the last ones spare), rot the rotations' (co, si), ph [n +
// 1] the phases and (1, 0); thread th of the vector, rows of 32 TW places.
template <typename R, int TW>
__device__ __forceinline__ void rows_step(typename Vec2<R>::T *X, const RowPlan &Q, int th, int bar,
                                          const typename Vec2<R>::T *rot, const typename Vec2<R>::T *ph) {
    typedef typename Vec2<R>::T R2;
    typedef Ar<R> A;
    constexpr int W = 32 * TW;
    const unsigned *ab = Q.ab + th;
    const unsigned short *id = Q.id + th;
    unsigned s0 = ab[0], y1 = id[W];
    R2 c0 = row_coef<R>(id[0], rot, ph);
    ab += W;
    id += 2 * W;
#pragma unroll 2
    for (int r = 0; r < Q.nrow; r++, ab += W, id += W) {
        R2 *pa = X + (s0 & 0xffff), *pb = X + (s0 >> 16);
        const R2 xa = *pa, xb = *pb;
        const unsigned s1 = ab[0], y2 = id[0];
        const R2 c1 = row_coef<R>(y1, rot, ph);
        R2 ya, yb;  // propagate.c:883-886
        ya.x = A::sub(A::mul(c0.x, xa.x), A::mul(c0.y, xb.y));
        ya.y = A::add(A::mul(c0.x, xa.y), A::mul(c0.y, xb.x));
        yb.x = A::sub(A::mul(c0.x, xb.x), A::mul(c0.y, xa.y));
        yb.y = A::add(A::mul(c0.x, xb.y), A::mul(c0.y, xa.x));
        *pa = ya;
        *pb = yb;
        rows_sync<TW>(bar);
        s0 = s1;
        y1 = y2;
        c0 = c1;
    }
}

// A vector's shared memory for rows_step: the state, the frame's phases and,
// with per-frame couplings, its rotations.
template <typename R> __host__ __device__ __forceinline__ size_t rows_vec_elems(int n, int K, bool rot_static, int TW) {
    return (size_t)(n + 32 * TW) + (n + 1) + (rot_static ? 0 : K);
}

// The step of a SinglesTab's Trotter tables through frame row fi; the vector's
// shared memory w (X first), rs the static rotations in shared memory.
template <typename R, int TW>
__device__ __forceinline__ void rows_singles_step(const SinglesTab &D, const RowPlan &Q, typename Vec2<R>::T *w,
                                                  const typename Vec2<R>::T *rs, int th, int bar, long fi) {
    typedef typename Vec2<R>::T R2;
    constexpr int W = 32 * TW;
    const int n = D.n;
    R2 *ph = w + n + W, *rot = ph + n + 1;
    const R2 *U = (const R2 *)D.U + fi * n;
    rows_sync<TW>(bar);
#pragma unroll 2
    for (int a = th; a < n; a += W) ph[a] = U[a];
    if (!D.rot_static) {
        const R2 *src = (const R2 *)D.rot + fi * D.K;
#pragma unroll 4
        for (int k = th; k < D.K; k += W) rot[k] = src[k];
        rs = rot;
    }
    rows_sync<TW>(bar);
    rows_step<R, TW>(w, Q, th, bar, rs, ph);
}

// A CTA of vectors on rows_singles_step: the schedule (where `stage`; Q then
// points to it) and the static rotations in shared memory, then the vectors' parts.
template <typename R, int TW>
__device__ __forceinline__ typename Vec2<R>::T *rows_setup(const SinglesTab &D, RowPlan &Q, bool stage,
                                                           unsigned char *smem, const typename Vec2<R>::T *&rs) {
    typedef typename Vec2<R>::T R2;
    constexpr int W = 32 * TW;
    const int vec = threadIdx.x / W, th = threadIdx.x % W, ne = W * (Q.nrow + 2);
    unsigned *as = (unsigned *)smem;
    unsigned short *is = (unsigned short *)(as + ne);
    R2 *rsh = (R2 *)(smem + (stage ? 6 * (size_t)ne : 0));
    const int Ks = D.rot_static ? D.K : 0;
    if (stage) {
        for (int e = threadIdx.x; e < ne; e += blockDim.x) {
            as[e] = Q.ab[e];
            is[e] = Q.id[e];
        }
        Q.ab = as;
        Q.id = is;
    }
    for (int k = threadIdx.x; k < Ks; k += blockDim.x) rsh[k] = ((const R2 *)D.rot)[k];
    R2 *w = rsh + Ks + vec * rows_vec_elems<R>(D.n, D.K, D.rot_static, TW);
    R2 z;
    z.x = z.y = 0;
    w[D.n + th] = z;  // the spare sites
    z.x = 1;
    if (th == 0) w[2 * D.n + W] = z;  // their phase
    __syncthreads();
    rs = rsh;
    return w;
}

// Launch shape: vectors per CTA and shared memory; 0 vectors if one does not fit.
struct RowShape {
    int vecs, stage;
    size_t bytes;
};
template <typename R> inline RowShape rows_shape(int n, int K, bool rot_static, int nrow, int TW, long vectors, int sms) {
    const size_t r2 = sizeof(typename Vec2<R>::T), ent = 192 * (size_t)TW * (nrow + 2), lim = 226 * 1024;
    const size_t per = r2 * rows_vec_elems<R>(n, K, rot_static, TW), rot = rot_static ? r2 * K : 0;
    const long want = std::min<long>(8 / TW, (vectors + sms - 1) / sms);
    RowShape s;
    // the schedule is staged where that leaves the wanted vectors their place, or
    // at least four of them (it is read again every step)
    s.stage = ent + rot + std::min<long>(want, 4) * per <= lim;
    const size_t base = rot + (s.stage ? ent : 0);
    s.vecs = (int)want;
    while (s.vecs > 0 && base + s.vecs * per > lim) s.vecs--;
    s.bytes = base + s.vecs * per;
    return s;
}

// Whether `vectors` go through the rows faster than a thread each (k_lin, k2d_gb1,
// k2d_gb3, k2d_se): until the vectors fill the threads, in FP32 about 860 operations
// per row and vector, 580 where the schedule is read from L2, in FP64 600 and 350.
// Measured: 16-site chain, 7422 vectors, 2.2 against 1.9 ms; the t3 vectors of 1500
// start points of 5 sites 4.0 against 0.73; FP64, 100 sites all coupled, 10 000 vectors
// (read from L2) 61 against 57, 3 sites, 1200 vectors of t3 0.34 against 0.31.
template <typename R> inline bool rows_pay(int n, int K, bool rot_static, int ts, const RowPlan &Q, long vectors, int sms) {
    if (!Q.ab) return false;
    const RowShape h = rows_shape<R>(n, K, rot_static, Q.nrow, 1, vectors, sms);
    const double most = sizeof(R) == 4 ? (h.stage ? 860 : 580) : (h.stage ? 600 : 350);
    return h.vecs > 0 && (double)vectors * Q.nrow < most * ts * (K + 2.0 * n);
}
