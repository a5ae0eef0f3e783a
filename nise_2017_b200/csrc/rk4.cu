// Linear absorption with the RK4 scheme (propagate_vec_RK4,
// propagate.c:261-373), a thread per site row.
//
// The reference walks the entries (a <= b) of the sparse Hamiltonian and adds
// each one's two contributions to the stage vectors, so the sum of row c runs
// over its neighbours (itself included) in ascending order, whatever the other
// rows do.  A thread that owns a row therefore performs the same operations in
// the same order from a list of the row's entries, and only the operand of a
// stage (c, c + k/2 or c + k) passes between threads.  The middle stages are
// evaluated in double as the reference's literal 0.5 promotes them; the
// promoted operand c + k/2 is formed once by its owner instead of once per
// entry.  The norms are summed in site order by every thread alike.
//
// A CTA takes one start point: its three polarisations share the frame's
// values and the row lists in shared memory, each on ceil(n/32) warps.  Bound
// by the latency of a row's chain (convert, add in double, convert: the
// reference's roundings), n links in each of two stages.  33 sites, 144 start
// points, RunTimes 64: 80.5 ms on a thread per vector (7 CTAs, every stage
// vector in shared memory), 2.4 ms now (144 CTAs).
#include "common.cuh"
#include "engine.h"
#include "schemes.cuh"

namespace {

// The operand of a middle stage, and its product with an entry.
template <typename R> struct Mid;
template <> struct Mid<float> {
    static __device__ __forceinline__ double op(float c, float k) { return __dadd_rn((double)c, __dmul_rn((double)k, 0.5)); }
    static __device__ __forceinline__ float plus(float acc, double h, double o) {
        return (float)__dadd_rn((double)acc, __dmul_rn(h, o));
    }
    static __device__ __forceinline__ float minus(float acc, double h, double o) {
        return (float)__dsub_rn((double)acc, __dmul_rn(h, o));
    }
};
template <> struct Mid<double> {
    static __device__ __forceinline__ double op(double c, double k) { return c + k * 0.5; }
    static __device__ __forceinline__ double plus(double acc, double h, double o) { return acc + h * o; }
    static __device__ __forceinline__ double minus(double acc, double h, double o) { return acc - h * o; }
};

// SM: the frame's values and the row lists in shared memory, else read from
// global memory.  WARP: one warp per vector (n <= 32).
template <typename R, bool SM, bool WARP>
__global__ void __launch_bounds__(960) k_abs_rk4_row(DevTraj T, Rk4Plan P, AbsJob J, double2 *resp, int G) {
    typedef typename Vec2<R>::T R2;
    typedef Ar<R> A;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = P.n, x = threadIdx.x / G, row = threadIdx.x % G, lane = threadIdx.x & 31;
    const bool act = row < n;
    double2 *bufs = (double2 *)smem_raw;         // [3][2][n] stage operands (R2 or double2 each)
    double2 *rs = bufs + 6 * n;                  // [3][n] response terms
    R *nrm = (R *)(rs + (WARP ? 0 : 3 * n));     // [3][2][n] norm terms
    R *vsh = nrm + 6 * n + (n & 1);              // [k] values of the frame
    uint32_t *tsh = (uint32_t *)(vsh + P.k + (P.k & 1));  // [slots][n] row lists
    double2 *b0 = bufs + 2 * x * n, *b1 = b0 + n;
    R *n0 = nrm + 2 * x * n, *n1 = n0 + n;
    auto sync = [&]() {
        if (WARP) __syncwarp();
        else __syncthreads();
    };
    if (SM)
        for (int e = threadIdx.x; e < P.slots * n; e += blockDim.x) tsh[e] = P.rows[e];
    const uint32_t *tab = (SM ? tsh : P.rows) + row;
    const int len = act ? P.len[row] : 0;
    const long ti = (long)(J.begin + blockIdx.x) * J.sample;
    R2 c;
    c.x = act ? (R)traj_mu(T, ti, x, row) : (R)0;
    c.y = 0;
    double2 *out = resp + (size_t)(3 * blockIdx.x + x) * J.tmax;
    for (int t1 = 0; t1 < J.tmax; t1++) {
        const long t = ti + t1;
        const R m = act ? (R)traj_mu(T, t, x, row) : (R)0;
        const double pr = act ? (double)A::mul(m, c.x) : 0.0, pi = act ? (double)A::mul(m, c.y) : 0.0;
        if (WARP) {
            const double2 z = resp_sum_warp(pr, pi, n);
            if (lane == 0) out[t1] = z;
        } else {  // a residue's sites in ascending order, then the residues (dot_mu)
            if (act) rs[x * n + row] = make_double2(pr, pi);
            __syncthreads();
            if (row < 32) {
                double sr = 0, si = 0;
                for (int i = row; i < n; i += 32) {
                    sr += rs[x * n + i].x;
                    si += rs[x * n + i].y;
                }
                const double2 z = resp_sum_warp(sr, si, n);
                if (lane == 0) out[t1] = z;
            }
        }
        if (t1 == J.tmax - 1) break;
        const R *val = (const R *)P.val + (size_t)(t - P.f0) * P.k;
        if (SM) {
            __syncthreads();
            for (int e = threadIdx.x; e < P.k; e += blockDim.x) vsh[e] = val[e];
            __syncthreads();
            val = vsh;
        }
        for (int sub = 0; sub < J.ts; sub++) {
            if (act) {
                *(R2 *)(b0 + row) = c;
                n0[row] = A::add(A::mul(c.x, c.x), A::mul(c.y, c.y));
            }
            sync();
            R2 k1, k2, k3, k4;
            auto outer = [&](const double2 *b) {  // first and last stage
                R2 k;
                k.x = k.y = 0;
#pragma unroll 4
                for (int q = 0; q < len; q++) {
                    const uint32_t e = tab[q * n];
                    const R h = val[e >> 10];
                    const R2 o = *(const R2 *)(b + (e & 1023));
                    k.x = A::add(k.x, A::mul(h, o.y));
                    k.y = A::sub(k.y, A::mul(h, o.x));
                }
                return k;
            };
            auto middle = [&](const double2 *b) {
                R2 k;
                k.x = k.y = 0;
#pragma unroll 4
                for (int q = 0; q < len; q++) {
                    const uint32_t e = tab[q * n];
                    const double h = (double)val[e >> 10];
                    const double2 o = b[e & 1023];
                    k.x = Mid<R>::plus(k.x, h, o.y);
                    k.y = Mid<R>::minus(k.y, h, o.x);
                }
                return k;
            };
            k1 = outer(b0);
            if (act) b1[row] = make_double2(Mid<R>::op(c.x, k1.x), Mid<R>::op(c.y, k1.y));
            sync();
            k2 = middle(b1);
            if (act) b0[row] = make_double2(Mid<R>::op(c.x, k2.x), Mid<R>::op(c.y, k2.y));
            sync();
            k3 = middle(b0);
            if (act) {
                R2 o;
                o.x = A::add(c.x, k3.x);
                o.y = A::add(c.y, k3.y);
                *(R2 *)(b1 + row) = o;
            }
            sync();
            k4 = outer(b1);
            c.x = Rk4Ops<R>::update(c.x, k1.x, k2.x, k3.x, k4.x);
            c.y = Rk4Ops<R>::update(c.y, k1.y, k2.y, k3.y, k4.y);
            if (act) n1[row] = A::add(A::mul(c.x, c.x), A::mul(c.y, c.y));
            sync();
            R norm = 0, nn = 0;  // find_norm, NISE_subs.c:125-133
#pragma unroll 8
            for (int i = 0; i < n; i++) {
                norm = A::add(norm, n0[i]);
                nn = A::add(nn, n1[i]);
            }
            if (norm != nn) {  // re_normalize, NISE_subs.c:136-148
                const R factor = (R)sqrt((double)(norm / nn));
                c.x = A::mul(c.x, factor);
                c.y = A::mul(c.y, factor);
            }
            sync();  // the norm terms are read before the next sub-step writes them
        }
    }
}

template <typename R>
int run_rk4_row(const DevTraj &T, const Rk4Plan &P, const AbsJob &J, double2 *resp, cudaStream_t s) {
    const int n = P.n, G = (n + 31) / 32 * 32;
    const bool warp = n <= 32;
    const size_t base = sizeof(double2) * (size_t)n * (warp ? 6 : 9) + sizeof(R) * (6 * (size_t)n + (n & 1));
    const size_t all = base + sizeof(R) * (size_t)(P.k + (P.k & 1)) + sizeof(uint32_t) * (size_t)P.slots * n;
    const bool sm = all <= 200 * 1024;
    auto kern = warp ? (sm ? k_abs_rk4_row<R, true, true> : k_abs_rk4_row<R, false, true>)
                     : (sm ? k_abs_rk4_row<R, true, false> : k_abs_rk4_row<R, false, false>);
    const size_t bytes = sm ? all : base;
    if (const int e = allow_smem(kern, bytes)) return e;
    kern<<<J.nsamp, 3 * G, bytes, s>>>(T, P, J, resp, G);
    return (int)cudaGetLastError();
}

// One step of caller vectors with their own packed Hamiltonians
// (nise_propagate): CTA per vector, a thread per row, the entries |H_ab| > cut
// and the diagonal in ascending order.  The values are in shared memory where
// they fit (VS).  60 vectors of 100 sites (the whole call): 19.6 ms with a thread
// per vector, 0.31 ms now.
template <typename R, bool VS>
__global__ void __launch_bounds__(1024) k_step_rk4_row(int n, float cut, const float *H, R *re, R *im, int ts, R fsub) {
    typedef typename Vec2<R>::T R2;
    typedef Ar<R> A;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *b0 = (double2 *)smem_raw, *b1 = b0 + n;
    R *n0 = (R *)(b1 + n), *n1 = n0 + n;
    float *hs = (float *)(n1 + n);
    const long nn2 = (long)n * (n + 1) / 2;
    const float *h = H + blockIdx.x * nn2;
    const int row = threadIdx.x;
    const bool act = row < n;
    if (VS) {
        for (long e = threadIdx.x; e < nn2; e += blockDim.x) hs[e] = h[e];
        h = hs;
    }
    R *pr = re + (size_t)blockIdx.x * n + row, *pi = im + (size_t)blockIdx.x * n + row;
    R2 c;
    c.x = act ? *pr : (R)0;
    c.y = act ? *pi : (R)0;
    // the entries of this row, in ascending neighbour order
    auto each = [&](auto f) {
        if (act)
            for (int r = 0; r < n; r++) {
                const float v = h[sindex(row, r, n)];
                if (fabsf(v) > cut || r == row) f(A::mul(fsub, (R)v), r);
            }
    };
    for (int sub = 0; sub < ts; sub++) {
        if (act) {
            *(R2 *)(b0 + row) = c;
            n0[row] = A::add(A::mul(c.x, c.x), A::mul(c.y, c.y));
        }
        __syncthreads();
        auto outer = [&](const double2 *b) {
            R2 k;
            k.x = k.y = 0;
            each([&](R v, int r) {
                const R2 o = *(const R2 *)(b + r);
                k.x = A::add(k.x, A::mul(v, o.y));
                k.y = A::sub(k.y, A::mul(v, o.x));
            });
            return k;
        };
        auto middle = [&](const double2 *b) {
            R2 k;
            k.x = k.y = 0;
            each([&](R v, int r) {
                const double2 o = b[r];
                k.x = Mid<R>::plus(k.x, (double)v, o.y);
                k.y = Mid<R>::minus(k.y, (double)v, o.x);
            });
            return k;
        };
        const R2 k1 = outer(b0);
        if (act) b1[row] = make_double2(Mid<R>::op(c.x, k1.x), Mid<R>::op(c.y, k1.y));
        __syncthreads();
        const R2 k2 = middle(b1);
        if (act) b0[row] = make_double2(Mid<R>::op(c.x, k2.x), Mid<R>::op(c.y, k2.y));
        __syncthreads();
        const R2 k3 = middle(b0);
        if (act) {
            R2 o;
            o.x = A::add(c.x, k3.x);
            o.y = A::add(c.y, k3.y);
            *(R2 *)(b1 + row) = o;
        }
        __syncthreads();
        const R2 k4 = outer(b1);
        c.x = Rk4Ops<R>::update(c.x, k1.x, k2.x, k3.x, k4.x);
        c.y = Rk4Ops<R>::update(c.y, k1.y, k2.y, k3.y, k4.y);
        if (act) n1[row] = A::add(A::mul(c.x, c.x), A::mul(c.y, c.y));
        __syncthreads();
        R norm = 0, nn = 0;
#pragma unroll 8
        for (int i = 0; i < n; i++) {
            norm = A::add(norm, n0[i]);
            nn = A::add(nn, n1[i]);
        }
        if (norm != nn) {
            const R factor = (R)sqrt((double)(norm / nn));
            c.x = A::mul(c.x, factor);
            c.y = A::mul(c.y, factor);
        }
        __syncthreads();
    }
    if (act) {
        *pr = c.x;
        *pi = c.y;
    }
}

template <typename R>
int run_step_rk4(int n, float cut, const float *H, R *re, R *im, int nvec, int ts, R fsub, cudaStream_t s) {
    const size_t base = sizeof(double2) * 2 * (size_t)n + sizeof(R) * 2 * n, all = base + sizeof(float) * (size_t)n * (n + 1) / 2;
    const bool vs = all <= 200 * 1024;
    auto kern = vs ? k_step_rk4_row<R, true> : k_step_rk4_row<R, false>;
    if (const int e = allow_smem(kern, vs ? all : base)) return e;
    kern<<<nvec, (n + 31) / 32 * 32, vs ? all : base, s>>>(n, cut, H, re, im, ts, fsub);
    return (int)cudaGetLastError();
}

}  // namespace

int launch_abs_rk4_row(int prec, const DevTraj &T, const Rk4Plan &P, const AbsJob &J, double2 *resp, cudaStream_t s) {
    if (J.nsamp <= 0) return 0;
    if (P.n > NISE_RK4_ROW_MAX_N) return (int)cudaErrorNotSupported;
    return prec == 0 ? run_rk4_row<float>(T, P, J, resp, s) : run_rk4_row<double>(T, P, J, resp, s);
}

int launch_step_rk4_row(int prec, int n, float cut, const float *H, void *re, void *im, int nvec, int ts, double fsub,
                        float fsub32, cudaStream_t s) {
    // below 8 sites a thread per vector where the vectors fill the threads: 2 sites, 50 000
    // vectors 0.50 against 0.34 ms, 5000 0.15 and 0.15; 5 sites 1.01 against 0.88 and 0.16
    // against 0.18
    if (n > 1024 || (n < 8 && nvec >= 1700 * n)) return (int)cudaErrorNotSupported;
    return prec == 0 ? run_step_rk4<float>(n, cut, H, (float *)re, (float *)im, nvec, ts, fsub32, s)
                     : run_step_rk4<double>(n, cut, H, (double *)re, (double *)im, nvec, ts, fsub, s);
}
