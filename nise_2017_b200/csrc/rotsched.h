// Schedule of the Trotter rotations of whole time steps (host only).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

// One rotation of a schedule: which one (q, an index into the coupling list),
// in which time step of the window (w), and whether that is the first or the
// last sub-step of its time step.
#define NISE_SCHED_Q(e) ((e) & 0xfffffu)
#define NISE_SCHED_W(e) (((e) >> 20) & 0xfu)
#define NISE_SCHED_FIRST(e) (((e) >> 30) & 1u)
#define NISE_SCHED_LAST(e) ((e) >> 31)
#define NISE_SCHED_NONE 0xfffffu
#define NISE_SCHED_MAX_K 0xfffff

// Rotation q's sites and its part in a sub-step: whether it is the first
// (PRE) or the last (POST) to touch its first (A) or second (B) site.  The
// half-step phase of a site belongs before its first and after its last
// rotation of every sub-step (propagate.c:870-894).
#define NISE_SCHED_A(p) ((p) & 0x3fffu)
#define NISE_SCHED_B(p) (((p) >> 14) & 0x3fffu)
#define NISE_SCHED_PRE_A(p) (((p) >> 28) & 1u)
#define NISE_SCHED_PRE_B(p) (((p) >> 29) & 1u)
#define NISE_SCHED_POST_A(p) (((p) >> 30) & 1u)
#define NISE_SCHED_POST_B(p) ((p) >> 31)
#define NISE_SCHED_MAX_N 0x3fff

// The rotations of `steps` time steps of `ts` sub-steps each, in rows of 32
// (one warp step each; NISE_SCHED_NONE fills a row up).  A rotation's level is
// 1 + the highest level of the earlier ones that share a site with it, across
// sub-step and step boundaries, so rotations that share a site keep the order
// of propagate.c:876-888 and a row's rotations are disjoint.  A coupling list
// with few disjoint neighbours (a chain: one rotation per level of a sub-step)
// runs its sub-steps as a wavefront: n + 2 (ts steps - 1) levels instead of
// n ts steps.  Returns the levels.
int nise_step_schedule(const std::vector<int2> &pairs, int n, int ts, int steps, std::vector<uint32_t> &rows);
// The packed sites and parts of every rotation; iso: the sites that no
// rotation touches.
void nise_schedule_parts(const std::vector<int2> &pairs, int n, std::vector<uint32_t> &parts, std::vector<int> &iso);

// Whole time steps as rows of `width` (a multiple of 32) independent operations
// of one kind, y_a = c x_a + i s x_b, y_b = c x_b + i s x_a: a rotation with its
// (co, si), or, with a = b, a site's half-step phase with its (cos, -sin) (the
// same float operations in the same order as propagate.c:870-873).  One step is
// `ts` times all phases, the rotations in order, all phases; every operation
// goes to the first row after the rows of the earlier operations on its sites
// that has room, so each site sees them in the reference's order.  ab = a | b <<
// 16; id = index into the rotation coefficients, or NISE_ROW_PHASE | site (six
// bytes a place: the schedule of a 500-site lattice fits shared memory).  Idle
// places rotate a spare site of their own, n + place, by the phase at index n, which the caller sets to (1, 0).  Two idle rows follow the last (a
// kernel reads two rows ahead).  Returns the number of rows without them.
#define NISE_ROW_PHASE 0x8000u
#define NISE_ROW_MAX 0x7fff  // couplings, and sites
int nise_row_schedule(const std::vector<int2> &pairs, int n, int ts, int width, std::vector<uint32_t> &ab,
                      std::vector<uint16_t> &id);
