// The decisions of `solve!` as device functions of the folded sums, shared by the
// single solve (solve_fast.cu) and the merged batch (batch.cu).
#pragma once

#include <cmath>

#include "cg_state.cuh"
#include "fused.cuh"

namespace tpa {

constexpr double kEps = 2.220446049250313e-16;

// std::max's choice, a NaN in second place included
__device__ __forceinline__ double std_max(double a, double b) { return a < b ? b : a; }

// roundoff floor of a residual from max |A||x| / V and max |b| / V
__host__ __device__ inline double roundoff_floor(double ax, double b) {
    const double m = ax < b ? b : ax;
    return 128 * kEps * (1.0 < m ? m : 1.0);
}

// What the solve was asked for (kernel parameters).
struct SolveAsk {
    double rtol, atol, cvol;  // cvol: volume of the ungauged component (0: none)
    double eta;               // refinement solve: reduction per run (0: one run to the target)
    int max_cycles, strict;   // strict: an incompatible right-hand side is an error
};

// target of a run from a residual of strong maximum linf
__device__ __forceinline__ double run_target(const SolveAsk& q, double target, double linf) {
    return q.eta > 0 ? std_max(target, q.eta * linf) : target;
}

__device__ __forceinline__ void start_run(CgState* c, double target, double rsum, int itmax, bool go) {
    c->target = target;
    c->rsum = rsum;
    c->itmax = itmax;
    c->iter = 0;
    c->fresh = 1;
    c->flags = go ? 0 : 8;
}

// After the first residual: the target, and the first run unless there is
// nothing to solve.  v: {sum_V r^2 / V, max |r| / V, max |A||x| / V, max |b| / V, sum r}.
__device__ __forceinline__ void after_first(const double (&v)[5], const SolveAsk& q, SolveState* S, CgState* c) {
    for (int k = 0; k < 4; ++k) S->init[k] = S->fin[k] = v[k];
    const double floor = roundoff_floor(v[2], v[3]);
    const double target = std_max(q.atol, std_max(q.rtol * std_max(v[1], kEps), floor));
    const bool go = S->ok && v[1] > target && q.max_cycles > 0;
    S->target = target;
    S->skip = go ? 0 : 1;
    S->niter = S->flags = S->total = 0;
    start_run(c, run_target(q, target, v[1]), v[4], q.max_cycles, go);
}

// After a run's true residual: its counts, and the state of a further run
// (which the host decides on).
__device__ __forceinline__ void after_run(const double (&v)[5], const SolveAsk& q, SolveState* S, CgState* c) {
    for (int k = 0; k < 4; ++k) S->fin[k] = v[k];
    S->niter = c->iter;
    S->flags = c->flags;
    S->total += c->iter;
    start_run(c, run_target(q, S->target, v[1]), v[4], q.max_cycles - S->total, true);
}

}  // namespace tpa
