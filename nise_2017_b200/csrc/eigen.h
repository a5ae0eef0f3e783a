// Batched FP64 eigendecomposition of per-frame Hamiltonians (eigen.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <algorithm>

#include "devtypes.h"

#define NISE_EIG_MAX_N 120

struct EigJob {
    DevTraj T;
    int n;
    int singleshift;
};

// Shared memory needed per frame.
size_t eig_smem_bytes(int n);
// Diagonalise the (shifted, cut) Hamiltonian of every frame in frames_dev:
// V[f][i][j] = component i of eigenvector j, w[f][j] ascending.
// n <= NISE_EIG_MAX_N (two FP64 n x n matrices in one CTA's shared memory).
int launch_eig(const EigJob &J, const long *frames_dev, long nframes, double *V, double *w, cudaStream_t s);

// Any n (eigen_large.cu): the Jacobi above up to NISE_EIG_MAX_N, else
// Householder tridiagonalisation + implicit QR (frames in parallel, one CTA
// each) with eig_any_ws_doubles(n, nframes) doubles of workspace A_ws and a
// status word set to 1 when a frame does not converge.  V's layout is
// private to the pair: pass it to launch_build_u_any.
size_t eig_any_ws_doubles(int n, long frames);
int launch_eig_any(const EigJob &J, const long *frames_dev, long nframes, double *V, double *w, double *A_ws,
                   int *status, cudaStream_t s);
// U[t] = V exp(-i w f) V^T (complex, working precision; |U|^2 <= thres
// dropped when truncate), for the layout of launch_eig_any.
int launch_build_u_any(int prec, const double *V, const double *w, long nfr, int n, double f, float thres,
                       int truncate, void *U, cudaStream_t s);

// exp(-i H f) of the frames [f0, f0 + nfr) without eigenvectors
// (propagators.cu), any n: U[t][a][c] in working precision (prec 0 FP32, 1
// FP64), exactly symmetric, |U|^2 <= thres dropped when truncate; ws holds
// propagator_ws_doubles(n) doubles for each of `ctas` CTAs (the results do not
// depend on their number).  *status (where not null) is set to 1 if a frame has a
// NaN or an infinity.
struct PropJob {
    DevTraj T;
    int n, singleshift, truncate;
    long f0, nfr;
    double f;
    float thres;
    int *status;
};
// Whether a job's propagators report such frames: above the size of the Jacobi,
// where the diagonalisation ended in an error; below, it passed them on.
inline bool propagators_report(int n) { return n > NISE_EIG_MAX_N; }
// CTAs for a job of that many frames whose workspaces take at most `room` bytes.
int propagator_ctas(int n, long frames, size_t room);
size_t propagator_ws_doubles(int n);
int launch_propagators(int prec, const PropJob &P, void *U, double *ws, int ctas, cudaStream_t s);
// The room a plan may hold, next to those of other jobs: what the eigenvectors
// and the QR workspace of 148 frames take, or 1 GB (up to 274 sites every SM has its
// CTAs, from 674 on 49 run); and what one call may take while it runs, if the device
// has it (300 frames of 512 sites, whole job: 30 ms against 60 in the held room).
inline size_t propagator_held(int n) { return std::max((size_t)1 << 30, (size_t)148 * 16 * n * n); }
const size_t kPropagatorRoom = (size_t)16 << 30;
