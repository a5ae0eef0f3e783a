// The exact one-step propagators U_t = exp(-i H_t f) of every frame, for
// Propagation Sparse and Diagonal with per-frame couplings or a truncating
// Threshold (propagate_vec_DIA, propagate_vec_DIA_S, propagate.c:60-258;
// time_evolution_mat, :1241-1299).
//
// The reference diagonalises every frame (ssyev_) and transforms the phases
// back; a propagator alone needs no eigenvectors.  With A = (H - c) f / 2^s, c
// the centre of the diagonal's range, the Taylor polynomials
//   cos A = sum_j (-1)^j X^j / (2j)!,  sin A = A sum_j (-1)^j X^j / (2j+1)!,
// X = A^2, are evaluated in FP64 from X, X^2 and X^3 (Paterson and Stockmeyer,
// SIAM J. Comput. 2 (1973) 60): 5 terms and 6 products while the Gershgorin
// bound of ||A|| is below 0.2 (remainder 0.2^12 / 12! = 9e-18), else 8 terms and
// 8 products up to 0.8 (0.8^18 / 18! = 3e-18), the power of two s bringing
// larger ones there; s doublings follow, and the phase exp(-i c f).  They double
// D = cos A - 1, D <- -2 S^2 and S <- 2 S + 2 S D: with cos itself an eigenvalue
// near c, where cos is near 1, has its error multiplied by 4 in every doubling, so
// that U U^H strays from 1 (80 sites and two 1500 cm^-1 away: 1e-13 after 4
// doublings, 2e-11 after 10; now 1e-15 and 5e-15, eigenvectors 3e-15).  What
// remains is the rounding of an eigenvalue, eps ||H f||, as with eigenvectors: the
// error of U against 64-bit mantissas is 1e-16 to 2e-15 up to 4 doublings
// (eigenvectors 1e-15 to 3e-15) and within 3 times the eigenvectors' beyond.  U is
// rounded to the working precision and truncated by the reference's test.
//
// One CTA per frame, frames dealt to as many CTAs as fit the SMs; the six
// matrices of a frame are in a workspace per CTA, which stays in L2 up to about 90
// sites (three CTAs per SM at 48 sites: 49 MB; two at 200: 570 MB).  All of them
// are polynomials in H, hence symmetric: only tiles on and above the diagonal
// are computed, the others mirrored, and both operands of a product are read
// along rows.  A thread holds 4 x 4 results; the tile is N / ceil(N / 64)
// rounded up to 4, so little of it is padding.  Bound by operand loads (L2 or
// device memory, then shared memory: 8 values for 16 multiply-adds) with two CTAs per SM to hide them: 48
// sites, 1987 frames 0.50 ms (Jacobi 4.8 ms); 200 sites, 595 frames 8.1 ms
// (Householder and QR 69.3 ms, then 1.4 ms for U).
#include <algorithm>

#include "common.cuh"
#include "eigen.h"
#include "engine.h"

namespace {

constexpr int kPuK = 16;    // rows of the operands staged per step
constexpr int kPuMat = 6;   // matrices of workspace per CTA

// c0 I + c1 M1 + c2 M2
struct Lin {
    double c0, c1, c2;
    const double *m1, *m2;
    __device__ __forceinline__ double at(int i, int j, int n) const {
        double v = i == j ? c0 : 0.0;
        if (m1) v = fma(c1, m1[(size_t)i * n + j], v);
        if (m2) v = fma(c2, m2[(size_t)i * n + j], v);
        return v;
    }
};

struct PuTile {
    int n, tx, nt, tile;  // tx x tx threads, nt x nt tiles of `tile` = 4 tx
    double (*As)[64], (*Bs)[64];
};

// out = A B + E for symmetric, commuting operands (B and E linear forms).
__device__ void pu_gemm(const PuTile &Q, double *out, const double *A, const Lin B, const Lin E) {
    const int n = Q.n, tid = threadIdx.x, cx = tid % Q.tx * 4, cy = tid / Q.tx * 4;
    const bool act = tid < Q.tx * Q.tx;
    for (int ti = 0; ti < Q.nt; ti++)
        for (int tj = ti; tj < Q.nt; tj++) {
            const int i0 = ti * Q.tile, j0 = tj * Q.tile;
            double acc[4][4] = {};
            for (int k0 = 0; k0 < n; k0 += kPuK) {
                __syncthreads();
                for (int e = tid; e < kPuK * Q.tile; e += blockDim.x) {
                    const int kk = e / Q.tile, q = e % Q.tile, k = k0 + kk;
                    Q.As[kk][q] = k < n && i0 + q < n ? A[(size_t)k * n + i0 + q] : 0.0;
                    Q.Bs[kk][q] = k < n && j0 + q < n ? B.at(k, j0 + q, n) : 0.0;
                }
                __syncthreads();
                if (!act) continue;
#pragma unroll
                for (int kk = 0; kk < kPuK; kk++) {
                    const double2 a0 = *(const double2 *)&Q.As[kk][cy], a1 = *(const double2 *)&Q.As[kk][cy + 2];
                    const double2 b0 = *(const double2 *)&Q.Bs[kk][cx], b1 = *(const double2 *)&Q.Bs[kk][cx + 2];
                    const double a[4] = {a0.x, a0.y, a1.x, a1.y}, b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
                    for (int p = 0; p < 4; p++)
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[p][q] = fma(a[p], b[q], acc[p][q]);
                }
            }
            if (act)
#pragma unroll
                for (int p = 0; p < 4; p++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int i = i0 + cy + p, j = j0 + cx + q;
                        if (i >= n || j >= n || i > j) continue;
                        const double v = acc[p][q] + E.at(i, j, n);
                        out[(size_t)i * n + j] = v;
                        out[(size_t)j * n + i] = v;
                    }
        }
    __syncthreads();
}

// The same with the next step's operands loaded while this one's are multiplied:
// with several tiles a third of the time was the wait for them (200 sites, 595
// frames: 10.8 -> 8.1 ms).  A single tile has few steps and other CTAs beside it, and
// is faster without (CD, 40 sites, FP64, whole job: 1.09 against 1.12 ms).
__device__ void pu_gemm_ahead(const PuTile &Q, double *out, const double *A, const Lin B, const Lin E) {
    constexpr int F = 6;  // elements a thread has in flight
    const int n = Q.n, tid = threadIdx.x, cx = tid % Q.tx * 4, cy = tid / Q.tx * 4;
    const bool act = tid < Q.tx * Q.tx;
    int pos[F];
    double fa[F], f1[F], f2[F];
#pragma unroll
    for (int u = 0; u < F; u++) {
        const int e = tid + u * blockDim.x;
        pos[u] = e < kPuK * Q.tile ? e / Q.tile << 8 | e % Q.tile : -1;
    }
    auto fetch = [&](int k0, int i0, int j0) {
#pragma unroll
        for (int u = 0; u < F; u++) {
            const int k = k0 + (pos[u] >> 8), q = pos[u] & 255;
            const bool in = pos[u] >= 0 && k < n;
            const size_t r = (size_t)k * n;
            fa[u] = in && i0 + q < n ? A[r + i0 + q] : 0.0;
            f1[u] = in && j0 + q < n && B.m1 ? B.m1[r + j0 + q] : 0.0;
            f2[u] = in && j0 + q < n && B.m2 ? B.m2[r + j0 + q] : 0.0;
        }
    };
    for (int ti = 0; ti < Q.nt; ti++)
        for (int tj = ti; tj < Q.nt; tj++) {
            const int i0 = ti * Q.tile, j0 = tj * Q.tile;
            double acc[4][4] = {};
            fetch(0, i0, j0);
            for (int k0 = 0; k0 < n; k0 += kPuK) {
                __syncthreads();
#pragma unroll
                for (int u = 0; u < F; u++)
                    if (pos[u] >= 0) {
                        const int kk = pos[u] >> 8, q = pos[u] & 255;
                        double v = k0 + kk == j0 + q && k0 + kk < n ? B.c0 : 0.0;
                        if (B.m1) v = fma(B.c1, f1[u], v);
                        if (B.m2) v = fma(B.c2, f2[u], v);
                        Q.As[kk][q] = fa[u];
                        Q.Bs[kk][q] = v;
                    }
                for (int e = tid + F * (int)blockDim.x; e < kPuK * Q.tile; e += blockDim.x) {
                    const int kk = e / Q.tile, q = e % Q.tile, k = k0 + kk;
                    Q.As[kk][q] = k < n && i0 + q < n ? A[(size_t)k * n + i0 + q] : 0.0;
                    Q.Bs[kk][q] = k < n && j0 + q < n ? B.at(k, j0 + q, n) : 0.0;
                }
                __syncthreads();
                if (k0 + kPuK < n) fetch(k0 + kPuK, i0, j0);
                if (!act) continue;
#pragma unroll
                for (int kk = 0; kk < kPuK; kk++) {
                    const double2 a0 = *(const double2 *)&Q.As[kk][cy], a1 = *(const double2 *)&Q.As[kk][cy + 2];
                    const double2 b0 = *(const double2 *)&Q.Bs[kk][cx], b1 = *(const double2 *)&Q.Bs[kk][cx + 2];
                    const double a[4] = {a0.x, a0.y, a1.x, a1.y}, b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
                    for (int p = 0; p < 4; p++)
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[p][q] = fma(a[p], b[q], acc[p][q]);
                }
            }
            if (act)
#pragma unroll
                for (int p = 0; p < 4; p++)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int i = i0 + cy + p, j = j0 + cx + q;
                        if (i >= n || j >= n || i > j) continue;
                        const double v = acc[p][q] + E.at(i, j, n);
                        out[(size_t)i * n + j] = v;
                        out[(size_t)j * n + i] = v;
                    }
        }
    __syncthreads();
}

// Largest value over the CTA (every thread gets it).
__device__ double pu_max(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) v = fmax(v, red[w]);
    return v;
}

template <typename R, bool AHEAD>
__global__ void __launch_bounds__(256, 2) k_propagators(PropJob P, int tx, int nt, typename Vec2<R>::T *U, double *ws) {
    typedef typename Vec2<R>::T R2;
    __shared__ __align__(16) double As[kPuK][64], Bs[kPuK][64];
    __shared__ double red[8];
    const int n = P.n, tid = threadIdx.x;
    const size_t nn = (size_t)n * n;
    const PuTile Q = {n, tx, nt, 4 * tx, As, Bs};
    double *A = ws + blockIdx.x * kPuMat * nn, *X = A + nn, *Y = X + nn, *Z = Y + nn, *C = Z + nn, *S = C + nn;
    const Lin zero = {0, 0, 0, nullptr, nullptr};
    const auto gemm = AHEAD ? pu_gemm_ahead : pu_gemm;
    for (long fr = blockIdx.x; fr < P.nfr; fr += gridDim.x) {
        const long t = P.f0 + fr;
        // H - c, its Gershgorin bound, and the scaling
        double hi = -1e300, lo = -1e300;
        for (int a = tid; a < n; a += blockDim.x) {
            const double h = (double)traj_diag(P.T, t, a, P.singleshift != 0);
            hi = fmax(hi, h);
            lo = fmax(lo, -h);
        }
        hi = pu_max(hi, red);
        lo = pu_max(lo, red);
        const double c = 0.5 * (hi - lo);
        for (int e = tid; e < n * n; e += blockDim.x) {
            const int a = e / n, b = e % n;
            A[e] = a == b ? (double)traj_diag(P.T, t, a, P.singleshift != 0) - c
                          : (double)traj_coupling(P.T, t, min(a, b), max(a, b));
        }
        __syncthreads();
        double r = 0;
        for (int a = tid; a < n; a += blockDim.x) {
            double s = 0;
            for (int b = 0; b < n; b++) s += fabs(A[(size_t)b * n + a]);
            if (P.status && !(s < HUGE_VAL)) *P.status = 1;  // (fmax passes over a NaN)
            r = fmax(r, s);
        }
        r = pu_max(r, red) * fabs(P.f);
        int s = 0;
        while (r > 0.8 && s < 60) {
            r *= 0.5;
            s++;
        }
        const double g = ldexp(P.f, -s);
        for (int e = tid; e < n * n; e += blockDim.x) A[e] *= g;
        __syncthreads();
        gemm(Q, X, A, {0, 1, 0, A, nullptr}, zero);
        gemm(Q, Y, X, {0, 1, 0, X, nullptr}, zero);
        gemm(Q, Z, X, {0, 1, 0, Y, nullptr}, zero);
        // reciprocal factorials with alternating signs: cc[j] = (-1)^j / (2j)!, sc[j] = (-1)^j / (2j+1)!
        double cc[9], sc[9];
        cc[0] = sc[0] = 1;
#pragma unroll
        for (int j = 1; j < 9; j++) {
            cc[j] = -cc[j - 1] / ((2.0 * j - 1) * (2.0 * j));
            sc[j] = -sc[j - 1] / ((2.0 * j) * (2.0 * j + 1));
        }
        double *Sn = r > 0.2 ? S : X, *f1 = Y, *f2 = Z;
        if (r > 0.2) {
            gemm(Q, S, Z, {cc[6], cc[7], cc[8], X, Y}, {cc[3], cc[4], cc[5], X, Y});
            gemm(Q, C, Z, {0, 1, 0, S, nullptr}, {0, cc[1], cc[2], X, Y});
            gemm(Q, S, Z, {sc[6], sc[7], sc[8], X, Y}, {sc[3], sc[4], sc[5], X, Y});
            // X is only read where it is written, by the same thread
            gemm(Q, X, Z, {0, 1, 0, S, nullptr}, {sc[0], sc[1], sc[2], X, Y});
            gemm(Q, Sn, A, {0, 1, 0, X, nullptr}, zero);
        } else {
            gemm(Q, C, Z, {cc[3], cc[4], cc[5], X, Y}, {0, cc[1], cc[2], X, Y});
            gemm(Q, S, Z, {sc[3], sc[4], sc[5], X, Y}, {sc[0], sc[1], sc[2], X, Y});
            gemm(Q, Sn, A, {0, 1, 0, S, nullptr}, zero);
        }
        double *Cn = C;  // cos A - 1
        for (int q = 0; q < s; q++) {
            gemm(Q, f1, Sn, {0, -2, 0, Sn, nullptr}, zero);
            gemm(Q, f2, Sn, {0, 2, 0, Cn, nullptr}, {0, 2, 0, Sn, nullptr});
            double *sw = Cn;
            Cn = f1;
            f1 = sw;
            sw = Sn;
            Sn = f2;
            f2 = sw;
        }
        double sp, cp;
        sincos(c * P.f, &sp, &cp);
        R2 *Uf = U + (size_t)fr * nn;
        for (int e = tid; e < n * n; e += blockDim.x) {
            const double co = Cn[e] + (e % (n + 1) == 0 ? 1.0 : 0.0), si = Sn[e];  // the diagonal: every n + 1
            R2 z;
            z.x = (R)(cp * co - sp * si);
            z.y = (R)(-(sp * co + cp * si));
            if (P.truncate) {  // propagate_vec_DIA_S keeps |U|^2 > Threshold, in the working precision
                bool keep;
                if (sizeof(R) == 4)
                    keep = __fadd_rn(__fmul_rn((float)z.x, (float)z.x), __fmul_rn((float)z.y, (float)z.y)) > P.thres;
                else
                    keep = (double)z.x * z.x + (double)z.y * z.y > (double)P.thres;
                if (!keep) z.x = z.y = (R)0;
            }
            Uf[e] = z;
        }
        __syncthreads();
    }
}

struct PuShape {
    int tx, nt, threads;
};
PuShape pu_shape(int n) {
    PuShape s;
    s.nt = (n + 63) / 64;
    s.tx = (n + 4 * s.nt - 1) / (4 * s.nt);
    s.threads = (s.tx * s.tx + 31) / 32 * 32;
    return s;
}

}  // namespace

// Resident CTAs by threads (128 registers each), and by the room for their
// workspaces.
int propagator_ctas(int n, long frames, size_t room) {
    const long per_sm = std::max(1, std::min(8, 512 / pu_shape(n).threads));
    return (int)std::max(1L, std::min(std::min(frames, per_sm * sm_count()), (long)(room / (sizeof(double) * propagator_ws_doubles(n)))));
}

size_t propagator_ws_doubles(int n) { return kPuMat * (size_t)n * n; }

int launch_propagators(int prec, const PropJob &P, void *U, double *ws, int ctas, cudaStream_t s) {
    if (P.nfr <= 0) return 0;
    const PuShape q = pu_shape(P.n);
    ctas = (int)std::min<long>(ctas, P.nfr);
    if (prec == 0)
        (q.nt > 1 ? k_propagators<float, true> : k_propagators<float, false>)<<<ctas, q.threads, 0, s>>>(P, q.tx, q.nt, (float2 *)U, ws);
    else
        (q.nt > 1 ? k_propagators<double, true> : k_propagators<double, false>)<<<ctas, q.threads, 0, s>>>(P, q.tx, q.nt, (double2 *)U, ws);
    return (int)cudaGetLastError();
}
