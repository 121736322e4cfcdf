// Device-resident scalars of the CG loop and of the solve around it.
#pragma once

namespace tpa {

// One Krylov run (solve_fused.cu).
struct CgState {
    double gamma, pAp, alpha, beta, pnorm2, strong_max, target, rsum, rnorm;
    int flags;  // 1 user exit, 2 zero curvature, 4 machine stop, 8 nothing to solve
    int iter, itmax;
    int fresh;  // the next r'z starts the run (gamma = r'z, p = z)
};

// flags that end a run in the middle of a loop body: the direction and the
// update of that body do nothing
constexpr int kCgHalt = 2 | 4 | 8;

// `solve!` around the runs (solve_fast.cu): every decision up to the end of the
// first run is taken on the device, and the host reads this once per run.
struct SolveState {
    double abs_b;                        // sum of magnitudes of b = V f
    double mb, mx, xm;                   // means removed from b, from the guess, from the iterate
    double init[4], fin[4];              // sum_V r^2 / V, max |r| / V, max |A||x| / V, max |b| / V
    double target;
    int ok;                              // the right-hand side is finite and compatible
    int skip;                            // the initial residual meets the target: no run
    int niter, flags, total;             // of the latest run; iterations of all runs
};

}  // namespace tpa
