// Single steps on caller Hamiltonians (nise_propagate), a CTA per vector: the
// Trotter scheme (propagate_vec_coupling_S, propagate.c:821-899) and the exact
// step (propagate_vec_DIA, propagate.c:60-125) by its Taylor series.
//
// The smallest call of the engine: what counts is the latency of one vector, so
// its work is spread over a CTA instead of one thread.
#include "common.cuh"
#include "engine.h"
#include "schemes.cuh"

namespace {

// Trotter with every pair in the list: the rotations with one sum a + b touch
// disjoint sites, and a site meets its rotations in ascending sums, which is
// their order in the list (propagate.c:876-888); so the sums 1 .. 2n - 3 are the
// levels, n/2 rotations wide.  The coefficients (a sine and a square root in
// double each) are formed once, by all threads.  16 sites, 3 vectors, 5
// sub-steps: 231 us on a thread per vector (which formed every coefficient in
// every sub-step), now 32 us.
template <typename R>
__global__ void __launch_bounds__(256) k_step_coupling_cta(int n, float cut, const float *H, R *re, R *im, int ts, R fsub) {
    typedef typename Vec2<R>::T R2;
    typedef Ar<R> A;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R2 *X = (R2 *)smem_raw, *U = X + n, *rot = U + n;  // rot: pairs a < b in list order
    const int tid = threadIdx.x, NT = blockDim.x;
    const float *h = H + (size_t)blockIdx.x * n * (n + 1) / 2;
    for (int a = tid; a < n; a += NT) {
        X[a].x = re[(size_t)blockIdx.x * n + a];
        X[a].y = im[(size_t)blockIdx.x * n + a];
        const double arg = 0.5 * (double)h[sindex(a, a, n)] * (double)fsub;
        U[a].x = (R)cos(arg);
        U[a].y = (R)(-sin(arg));
    }
    const int np = n * (n - 1) / 2;
    for (int e = tid; e < np; e += NT) {
        int a = 0, rem = e;
        while (rem >= n - 1 - a) { rem -= n - 1 - a; a++; }
        const float j = h[sindex(a, a + 1 + rem, n)];
        R2 cs;
        cs.x = 2;  // not in the list
        cs.y = 0;
        if (fabsf(j) > cut) cs = Cst<R>::rot(j, fsub, cut);
        rot[e] = cs;
    }
    auto sync = [&]() {
        if (NT == 32) __syncwarp();
        else __syncthreads();
    };
    sync();
    auto phase = [&]() {
        for (int a = tid; a < n; a += NT) {
            const R2 z = X[a], u = U[a];
            R2 o;
            o.x = A::sub(A::mul(z.x, u.x), A::mul(z.y, u.y));
            o.y = A::add(A::mul(z.y, u.x), A::mul(z.x, u.y));
            X[a] = o;
        }
        sync();
    };
    for (int sub = 0; sub < ts; sub++) {
        phase();
        for (int s = 1; s <= 2 * n - 3; s++) {
            for (int a = max(0, s - n + 1) + tid; 2 * a < s; a += NT) {
                const int b = s - a;
                const R2 cs = rot[a * (2 * n - a - 1) / 2 + b - a - 1];
                if (cs.x > (R)1) continue;
                const R2 xa = X[a], xb = X[b];
                R2 ya, yb;
                ya.x = A::sub(A::mul(cs.x, xa.x), A::mul(cs.y, xb.y));
                ya.y = A::add(A::mul(cs.x, xa.y), A::mul(cs.y, xb.x));
                yb.x = A::sub(A::mul(cs.x, xb.x), A::mul(cs.y, xa.y));
                yb.y = A::add(A::mul(cs.x, xb.y), A::mul(cs.y, xa.x));
                X[a] = ya;
                X[b] = yb;
            }
            sync();
        }
        phase();
    }
    for (int a = tid; a < n; a += NT) {
        re[(size_t)blockIdx.x * n + a] = X[a].x;
        im[(size_t)blockIdx.x * n + a] = X[a].y;
    }
}

// The exact step: a thread per row, the products of a term in site order (as a
// thread per vector adds them), H in shared memory where it fits (HS).
template <typename R, bool HS>
__global__ void __launch_bounds__(1024) k_step_taylor_cta(int n, const float *H, R *re, R *im, double f) {
    typedef typename Vec2<R>::T R2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[32];
    R2 *cur = (R2 *)smem_raw, *nxt = cur + n;
    float *hs = (float *)(nxt + n);
    const long nn2 = (long)n * (n + 1) / 2;
    const float *h = H + blockIdx.x * nn2;
    const int a = threadIdx.x;
    const bool act = a < n;
    if (HS) {
        for (long e = threadIdx.x; e < nn2; e += blockDim.x) hs[e] = h[e];
        h = hs;
        __syncthreads();
    }
    R *pr = re + (size_t)blockIdx.x * n + a, *pi = im + (size_t)blockIdx.x * n + a;
    double bound = 0;
    if (act)
        for (int b = 0; b < n; b++) bound += fabs((double)h[sindex(a, b, n)]);
    for (int o = 16; o > 0; o >>= 1) bound = fmax(bound, __shfl_xor_sync(0xffffffffu, bound, o));
    if ((a & 31) == 0) red[a >> 5] = bound;
    R2 acc;
    acc.x = act ? *pr : (R)0;
    acc.y = act ? *pi : (R)0;
    if (act) cur[a] = acc;
    __syncthreads();
    bound = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) bound = fmax(bound, red[w]);
    const double bnd = fabs(f) * bound, tol = sizeof(R) == 4 ? 1e-12 : 1e-18;
    double term = exp(bnd);
    int K;
    for (K = 0; K < 80; K++) {
        term *= bnd / (K + 1);
        if (term <= tol) break;
    }
    for (int k = 1; k <= K; k++) {
        const R c = (R)(f / k);
        if (act) {
            R yr = 0, yi = 0;
#pragma unroll 4
            for (int b = 0; b < n; b++) {
                const R w = (R)h[sindex(a, b, n)];
                const R2 z = cur[b];
                yr += w * z.x;
                yi += w * z.y;
            }
            R2 nz;
            nz.x = c * yi;
            nz.y = -c * yr;
            nxt[a] = nz;
            acc.x += nz.x;
            acc.y += nz.y;
        }
        __syncthreads();
        R2 *tmp = cur;
        cur = nxt;
        nxt = tmp;
    }
    if (act) {
        *pr = acc.x;
        *pi = acc.y;
    }
}

template <typename R>
int run_coupling(int n, float cut, const float *H, R *re, R *im, int nvec, int ts, R fsub, cudaStream_t s) {
    const size_t bytes = sizeof(typename Vec2<R>::T) * (2 * (size_t)n + (size_t)n * (n - 1) / 2);
    // a thread per vector again where the vectors fill the threads: whole calls of 2, 8
    // and 16 sites with 50 000 vectors 0.39, 1.51 and 3.78 ms against 0.33, 1.32 and 3.66,
    // with 10 000 0.12, 0.38 and 0.87 against 0.11, 0.39 and 1.04
    if (bytes > 220 * 1024 || nvec >= 2500L * n) return (int)cudaErrorNotSupported;
    if (const int e = allow_smem(k_step_coupling_cta<R>, bytes)) return e;
    k_step_coupling_cta<R><<<nvec, (n + 63) / 64 * 32, bytes, s>>>(n, cut, H, re, im, ts, fsub);
    return (int)cudaGetLastError();
}

template <typename R>
int run_taylor(int n, const float *H, R *re, R *im, int nvec, double f, cudaStream_t s) {
    const size_t base = sizeof(typename Vec2<R>::T) * 2 * (size_t)n, all = base + sizeof(float) * (size_t)n * (n + 1) / 2;
    const bool hs = all <= 200 * 1024;
    auto kern = hs ? k_step_taylor_cta<R, true> : k_step_taylor_cta<R, false>;
    if (const int e = allow_smem(kern, hs ? all : base)) return e;
    kern<<<nvec, (n + 31) / 32 * 32, hs ? all : base, s>>>(n, H, re, im, f);
    return (int)cudaGetLastError();
}

}  // namespace

int launch_step_coupling_cta(int prec, int n, float cut, const float *H, void *re, void *im, int nvec, int ts,
                             double fsub, float fsub32, cudaStream_t s) {
    return prec == 0 ? run_coupling<float>(n, cut, H, (float *)re, (float *)im, nvec, ts, fsub32, s)
                     : run_coupling<double>(n, cut, H, (double *)re, (double *)im, nvec, ts, fsub, s);
}

int launch_step_taylor_cta(int prec, int n, const float *H, void *re, void *im, int nvec, double f, cudaStream_t s) {
    // below 8 sites a thread per vector where the vectors fill the threads: 5 sites, 50 000
    // vectors 0.84 against 0.76 ms, 10 000 0.20 and 0.20; 8 sites are no slower here
    if (n > 1024 || (n < 8 && nvec >= 2500 * n)) return (int)cudaErrorNotSupported;
    return prec == 0 ? run_taylor<float>(n, H, (float *)re, (float *)im, nvec, f, s)
                     : run_taylor<double>(n, H, (double *)re, (double *)im, nvec, f, s);
}
