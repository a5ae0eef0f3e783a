// One Trotter time step of a vector on a warp, from the rows of
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
__device__ __forceinline__ typename Vec2<R>::T row_coef(uint32_t y, const typename Vec2<R>::T *rot,
                                                        const typename Vec2<R>::T *ph) {
    return ((y & NISE_ROW_PHASE) ? ph : rot)[y & ~NISE_ROW_PHASE];
}

// X [n + 32] state (the last 32 spare), rot the rotations' (co, si), ph [n + 1]
// the phases and (1, 0); I entries per lane and row.
template <typename R, int I>
__device__ __forceinline__ void rows_step(typename Vec2<R>::T *X, const uint2 *rows, int nrow, int lane,
                                          const typename Vec2<R>::T *rot, const typename Vec2<R>::T *ph) {
    typedef typename Vec2<R>::T R2;
    typedef Ar<R> A;
    uint2 e0[I], e1[I];
    R2 c0[I];
#pragma unroll
    for (int i = 0; i < I; i++) {
        e0[i] = rows[32 * i + lane];
        e1[i] = rows[32 * (I + i) + lane];
        c0[i] = row_coef<R>(e0[i].y, rot, ph);
    }
    const uint2 *next = rows + 64 * I + lane;
#pragma unroll 2
    for (int r = 0; r < nrow; r++, next += 32 * I) {
        R2 xa[I], xb[I], c1[I];
#pragma unroll
        for (int i = 0; i < I; i++) {
            xa[i] = X[e0[i].x & 0xffff];
            xb[i] = X[e0[i].x >> 16];
        }
        uint2 e2[I];
#pragma unroll
        for (int i = 0; i < I; i++) {
            e2[i] = next[32 * i];
            c1[i] = row_coef<R>(e1[i].y, rot, ph);
        }
#pragma unroll
        for (int i = 0; i < I; i++) {  // propagate.c:883-886
            R2 ya, yb;
            ya.x = A::sub(A::mul(c0[i].x, xa[i].x), A::mul(c0[i].y, xb[i].y));
            ya.y = A::add(A::mul(c0[i].x, xa[i].y), A::mul(c0[i].y, xb[i].x));
            yb.x = A::sub(A::mul(c0[i].x, xb[i].x), A::mul(c0[i].y, xa[i].y));
            yb.y = A::add(A::mul(c0[i].x, xb[i].y), A::mul(c0[i].y, xa[i].x));
            X[e0[i].x & 0xffff] = ya;
            X[e0[i].x >> 16] = yb;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < I; i++) {
            e0[i] = e1[i];
            e1[i] = e2[i];
            c0[i] = c1[i];
        }
    }
}

// A warp's shared memory for rows_step: the state, the frame's phases and,
// with per-frame couplings, its rotations.
template <typename R> __host__ __device__ __forceinline__ size_t rows_warp_elems(int n, int K, bool rot_static) {
    return (size_t)(n + 32) + (n + 1) + (rot_static ? 0 : K);
}

// The step of a SinglesTab's Trotter tables through frame row fi; the warp's
// shared memory w (X first), rs the static rotations in shared memory.
template <typename R>
__device__ __forceinline__ void rows_singles_step(const SinglesTab &D, const uint2 *rows, int nrow, typename Vec2<R>::T *w,
                                                  const typename Vec2<R>::T *rs, int lane, long fi) {
    typedef typename Vec2<R>::T R2;
    const int n = D.n;
    R2 *ph = w + n + 32, *rot = ph + n + 1;
    const R2 *U = (const R2 *)D.U + fi * n;
    __syncwarp();
#pragma unroll 2
    for (int a = lane; a < n; a += 32) ph[a] = U[a];
    if (!D.rot_static) {
        const R2 *src = (const R2 *)D.rot + fi * D.K;
#pragma unroll 4
        for (int k = lane; k < D.K; k += 32) rot[k] = src[k];
        rs = rot;
    }
    __syncwarp();
    rows_step<R, 1>(w, rows, nrow, lane, rs, ph);
}

// A CTA of warps on rows_singles_step: the schedule (STAGE) and the static
// rotations in shared memory, then the warps' parts.
template <typename R>
__device__ __forceinline__ typename Vec2<R>::T *rows_setup(const SinglesTab &D, const RowPlan &Q, bool stage,
                                                           unsigned char *smem, const uint2 *&rows,
                                                           const typename Vec2<R>::T *&rs) {
    typedef typename Vec2<R>::T R2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ne = 32 * (Q.nrow + 2);
    uint2 *es = (uint2 *)smem;
    R2 *rsh = (R2 *)(smem + (stage ? sizeof(uint2) * (size_t)ne : 0));
    const int Ks = D.rot_static ? D.K : 0;
    if (stage)
        for (int e = threadIdx.x; e < ne; e += blockDim.x) es[e] = Q.rows[e];
    for (int k = threadIdx.x; k < Ks; k += blockDim.x) rsh[k] = ((const R2 *)D.rot)[k];
    R2 *w = rsh + Ks + warp * rows_warp_elems<R>(D.n, D.K, D.rot_static);
    R2 z;
    z.x = z.y = 0;
    w[D.n + lane] = z;  // the spare sites
    z.x = 1;
    if (lane == 0) w[2 * D.n + 32] = z;  // their phase
    __syncthreads();
    rows = stage ? es : Q.rows;
    rs = rsh;
    return w;
}

// Launch shape: warps per CTA and shared memory; 0 warps if a vector does not fit.
struct RowShape {
    int warps, stage;
    size_t bytes;
};
template <typename R> inline RowShape rows_shape(int n, int K, bool rot_static, int nrow, long vectors, int sms) {
    const size_t r2 = sizeof(typename Vec2<R>::T), ent = sizeof(uint2) * 32 * (size_t)(nrow + 2);
    const size_t per = r2 * rows_warp_elems<R>(n, K, rot_static), rot = rot_static ? r2 * K : 0;
    RowShape s;
    s.stage = ent + rot + per <= 220 * 1024 && ent <= 128 * 1024;
    const size_t base = rot + (s.stage ? ent : 0);
    s.warps = (int)std::min<long>(8, (vectors + sms - 1) / sms);
    while (s.warps > 0 && base + s.warps * per > 220 * 1024) s.warps--;
    s.bytes = base + s.warps * per;
    return s;
}
