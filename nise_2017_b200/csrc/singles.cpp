// Coefficient tables of the singles propagation schemes over the frames of
// one job, shared by the 2D and linear-technique drivers.
//
// The reference rebuilds the propagator of a frame for every vector it
// propagates through that frame (propagate_vector, propagate.c:20-39).  Here
// each frame's coefficients are computed once per job and read by every
// vector: Trotter half phases and rotation coefficients (k_prep_trotter), the
// RK4 Hamiltonian entries (k_prep_rk4), or, for Sparse/Diagonal, the one-step
// propagator exp(-i H f) (propagators.cu).  With doubles, that route also builds
// the truncated sub-step propagator of time_evolution_mat
// (propagate.c:1241-1299).
#include <algorithm>
#include <vector>

#include "eigen.h"
#include "engine.h"
#include "nise_internal.h"
#include "rotsched.h"

int nise_singles_tables(nise_ctx *c, const DevTraj &T, long fmin, long nf, int singleshift, bool doubles_u,
                        SinglesTab &S, SinglesBufs &B) {
    const nise_params &p = c->p;
    const int N = c->n, prec = p.precision;
    const size_t rsz = prec == NISE_FP32 ? sizeof(float) : sizeof(double), r2 = 2 * rsz;
    int rc;
    std::vector<int2> pairs;
    if ((rc = nise_pattern(c, fmin, nf, pairs))) return rc;
    const int K = (int)pairs.size();
    // segments of one first site and one warp (b >> 5) of second sites, for
    // the doubles kernel that shares a vector between two warps
    std::vector<int4> segs;
    for (int k = 0; k < K;) {
        const int a = pairs[k].x, w = pairs[k].y >> 5, k0 = k;
        while (k < K && pairs[k].x == a && (pairs[k].y >> 5) == w) k++;
        segs.push_back(make_int4(a, k0, k, w));
    }
    if (segs.empty()) segs.push_back(make_int4(0, 0, 0, 0));
    pairs.push_back(make_int2(0, 0));  // one record past the last: read ahead without a bound check
    if ((rc = B.pairs.upload(c, pairs)) || (rc = B.segs.upload(c, segs))) return rc;
    S.n = N;
    S.ts = p.ts;
    S.prop = p.propagation;
    S.f0 = fmin;
    S.pairs = B.pairs.p;
    S.K = K;
    S.segs = B.segs.p;
    S.nsegs = K ? (int)segs.size() : 0;
    S.U = S.rot = S.rkval = S.Ud = nullptr;
    S.ent = nullptr;
    S.Kr = 0;
    S.rot_static = p.hamiltonian == NISE_HAM_COUPLING;
    B.Us = nullptr;
    if (p.propagation == NISE_PROP_COUPLING) {
        TrotterPlan P;
        P.n = N; P.k = S.K; P.pairs = B.pairs.p; P.f0 = fmin; P.nf = nf;
        P.rot_static = S.rot_static;
        P.singleshift = singleshift;
        if ((rc = B.U.alloc(c, r2 * (size_t)nf * N))) return rc;
        if ((rc = B.rot.alloc(c, r2 * (size_t)(P.rot_static ? 1 : nf) * (P.k ? P.k : 1)))) return rc;
        P.U = B.U.p;
        P.rot = B.rot.p;
        if ((rc = nise_cuda(c, launch_prep_trotter(prec, T, P, nise_f64(p, 1, p.ts), nise_f32(p, 1, p.ts), c->stream),
                            "Trotter prep")))
            return rc;
        c->launches += 1 + P.rot_static;
        S.U = B.U.p;
        S.rot = B.rot.p;
        // (a single coupling leaves nothing to put side by side)
        if (K >= 2 && N + 64 <= NISE_ROW_MAX && K <= NISE_ROW_MAX && p.ts >= 1) {
            std::vector<uint32_t> ab;
            std::vector<uint16_t> id;
            pairs.pop_back();
            B.row.nrow = nise_row_schedule(pairs, N, p.ts, 32, ab, id);
            if ((rc = B.row_ab.upload(c, ab)) || (rc = B.row_id.upload(c, id))) return rc;
            B.row.ab = B.row_ab.p;
            B.row.id = B.row_id.p;
        }
    } else if (p.propagation == NISE_PROP_SPARSE || p.propagation == NISE_PROP_DIAGONAL) {
        // propagate_vector's Sparse scheme (DIA, or DIA_S when 0 < Threshold
        // <= 1) and time_evolution_mat's truncated sub-step propagator for the
        // doubles (Threshold always applied); Diagonal is the untruncated
        // exact propagator.
        if (N > 1024)
            return nise_fail(c, NISE_ERR_UNSUPPORTED, "Propagation Sparse/Diagonal on per-frame tables is limited to "
                             "1024 sites");
        const float thr = p.propagation == NISE_PROP_DIAGONAL ? 0.0f : c->thres;
        const bool trunc_singles = thr != 0 && !(thr > 1);
        DevBuf<double> ws;
        DevBuf<int> status;
        if (propagators_report(N)) {
            if ((rc = status.alloc(c, 1))) return rc;
            cudaMemsetAsync(status.p, 0, sizeof(int), c->stream);
        }
        if ((rc = B.U.alloc(c, r2 * (size_t)nf * N * N))) return rc;
        if (doubles_u && (rc = B.rot.alloc(c, r2 * (size_t)nf * N * N))) return rc;
        int ctas = propagator_ctas(N, nf, kPropagatorRoom);
        if (!ws.try_alloc(c, ctas * propagator_ws_doubles(N))) {
            ctas = propagator_ctas(N, nf, propagator_held(N));
            if ((rc = ws.alloc(c, ctas * propagator_ws_doubles(N)))) return rc;
        }
        const int pr = prec == NISE_FP32 ? 0 : 1;
        PropJob PJ;
        PJ.T = T;
        PJ.n = N;
        PJ.singleshift = singleshift;
        PJ.f0 = fmin;
        PJ.nfr = nf;
        PJ.thres = thr;
        PJ.status = status.p;
        PJ.truncate = trunc_singles;
        PJ.f = prec == NISE_FP32 ? (double)nise_f32(p, 1, 1) : nise_f64(p, 1, 1);
        if ((rc = nise_cuda(c, launch_propagators(pr, PJ, B.U.p, ws.p, ctas, c->stream), "propagator build"))) return rc;
        c->launches++;
        if (doubles_u) {
            PJ.truncate = 1;
            PJ.f = prec == NISE_FP32 ? (double)nise_f32(p, 1, p.ts) : nise_f64(p, 1, p.ts);
            if ((rc = nise_cuda(c, launch_propagators(pr, PJ, B.rot.p, ws.p, ctas, c->stream), "doubles propagator build")))
                return rc;
            c->launches++;
        }
        if (status.p) {
            int bad = 0;
            if ((rc = nise_cuda(c, (int)cudaMemcpyAsync(&bad, status.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream),
                                "propagator status")) ||
                (rc = nise_cuda(c, (int)cudaStreamSynchronize(c->stream), "propagators")))
                return rc;
            if (bad) return nise_fail(c, NISE_ERR_DEVICE, NISE_NOT_FINITE);
        }
        S.Ud = B.U.p;
        if (doubles_u) B.Us = B.rot.p;
    } else {
        std::vector<int2> ent;
        size_t q = 0;
        for (int a = 0; a < N; a++) {
            ent.push_back(make_int2(a, a));
            while (q < (size_t)K && pairs[q].x == a) ent.push_back(pairs[q++]);
        }
        if ((rc = B.ent.upload(c, ent))) return rc;
        Rk4Plan P;
        P.n = N; P.k = (int)ent.size(); P.entries = B.ent.p; P.f0 = fmin; P.nf = nf; P.singleshift = singleshift;
        if ((rc = B.rkval.alloc(c, rsz * (size_t)nf * P.k))) return rc;
        P.val = B.rkval.p;
        if ((rc = nise_cuda(c, launch_prep_rk4(prec, T, P, nise_f64(p, 1, p.ts), nise_f32(p, 1, p.ts), c->stream),
                            "RK4 prep")))
            return rc;
        c->launches++;
        S.ent = B.ent.p;
        S.Kr = P.k;
        S.rkval = B.rkval.p;
    }
    return NISE_OK;
}
