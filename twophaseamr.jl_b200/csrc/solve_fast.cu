// `solve!` around the graph-captured CG loop, with its set-up and checks fused
// into finest-level passes (default cycle, at most one ungauged component).
//
// The steps are those of src/solvers/multigrid/elliptic_solver.jl:628-675
// (ronaldremmerswaal/TwoPhaseAMR.jl): b = V f with covered cells zeroed, the
// component projection of b (`_project_component_rhs!`, :153-190), the gauge of
// the initial guess, the initial norms and target (`_solve_krylov_with_stats!`,
// :550-612, with the roundoff floor of cycles.jl:108-206), Krylov runs with
// restarts from the true residual (`_run_krylov_reliably!`, :487-526) and the
// final gauge.
//
// `k_prep` folds the three sums the projection and the gauge need; `k_pres`
// applies them and evaluates the residual, its norms and both inputs of the
// roundoff floor in one pass.  The CTA that folds them also takes the decision
// that follows (means, target, whether there is anything to solve, the state of
// the run), so a solve is one chain of launches that the host reads once, at
// the end of the first run: prep, pres, the CG graph, the iterate's mean, pres.
// Reading every decision on the host took six synchronizations of 8-15 us each,
// and the run started with a residual pass of its own.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "cg_state.cuh"
#include "device.cuh"
#include "launch.cuh"
#include "solve_state.cuh"

namespace tpa {
namespace {

constexpr int kGrid = 1184;  // 8 CTAs on each of 148 SMs
constexpr int kCPrep = 8, kCPres = 9, kCMean = 10;

// N values folded over the grid, value k in partial[k gridDim.x ..)
template <int N, int WARP = kWarpFold, typename F>
__device__ __forceinline__ void publish_fold(const double (&v)[N], unsigned max_mask, double* partial,
                                             unsigned* counter, F done) {
    double* p[N];
    for (int k = 0; k < N; ++k) p[k] = partial + k * gridDim.x;
    fold_blocks<N, WARP>(v, max_mask, p, counter, blockIdx.x, 0, gridDim.x, done);
}

// sums of b = V f, |b| and V x0 over cells with V > 0; the means to remove.
// vol null: every cell's volume is vol0.
__global__ void k_prep(int n, const double* rhs, const double* xin,
                       const double* __restrict__ vol, double vol0, SolveAsk q, double* partial, unsigned* counter,
                       SolveState* S) {
    pdl_entry();
    double v[3] = {0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double V = vol ? vol[i] : vol0;
        const double bi = V > 0 ? rhs[i] * V : 0.0;
        const double xi = V > 0 ? xin[i] : 0.0;
        v[0] += bi;
        v[1] += fabs(bi);
        v[2] += V * xi;
    }
    // in the order of the plain solve's sums: the removed mean is often rounding alone
    publish_fold<3, 0>(v, 0u, partial, counter, [&](const double (&t)[3]) {
        S->abs_b = t[1];
        const bool comp = q.cvol != 0;
        S->mb = comp ? t[0] / q.cvol : 0.0;
        S->mx = comp ? t[2] / q.cvol : 0.0;
        S->xm = 0;
        // a non-finite right-hand side value makes sum |b| non-finite
        S->ok = isfinite(t[1]) && !(q.strict && comp && fabs(t[0]) > 256 * kEps * std_max(1.0, t[1]));
    });
}

// Vectors of a residual pass.  First: b = V f - V mb and x = x_in - mx (0 where
// V = 0) are formed from the caller's rhs and guess and stored; else b and x
// are the solve's and x - xm goes to the caller's array.
struct PresIo {
    const double* rhs;  // the caller's (first pass)
    const double* xin;  // the guess (first) or the iterate
    double* b;
    double* xout;       // the solve's iterate (first) or the caller's solution
    double* r;
};

// r = b - A x with the norms.  A x is summed as sum_j a_ij (x_j - x_i) (+ bdiag_i
// x_i at open sides): the rows sum to that conductance (the area-weighted jump
// maps constants to zero), and this form rounds at
// the level of the face fluxes, as the factorized action of elliptic.jl:
// 1125-1180 does, not at the level of a_ii x_i.  The projection step relies on
// it: dt max |div u| after the update equals the final residual over 1/dt^2 to
// a few ulps only when both are evaluated from face differences.
template <bool First>
__global__ void k_pres(LevelView<double> A, PresIo io, int masked, SolveAsk q, double* partial, unsigned* counter,
                       SolveState* S, CgState* c) {
    pdl_entry();
    const double m = First ? S->mx : S->xm, mb = First ? S->mb : 0.0;
    const bool store = First || S->ok;
    const double* x0 = io.xin;
    double v[5] = {0, 0, 0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n; i += gridDim.x * blockDim.x) {
        const double V = A.vol[i];
        double bi;
        if (First) {
            bi = V > 0 ? io.rhs[i] * V : 0.0;
            if (mb != 0.0 && V > 0) bi -= V * mb;
            io.b[i] = bi;
        } else {
            bi = io.b[i];
        }
        const double xi = V > 0 ? x0[i] - m : 0.0;
        double acc = 0, aacc = 0;
        for (int k = A.rp[i]; k < A.rp[i + 1]; ++k) {
            const int j = A.ci[k];
            const double xj = (!masked || A.vol[j] > 0) ? x0[j] - m : 0.0;
            acc += A.val[k] * (xj - xi);
            aacc += fabs(A.val[k]) * fabs(xj);
        }
        if (A.bdiag) acc += A.bdiag[i] * xi;  // rows at open sides do not sum to zero
        if (store) io.xout[i] = xi;
        const double ri = bi - acc;
        io.r[i] = ri;
        v[4] += ri;
        if (V > 0) {
            v[0] += ri * ri / V;
            const double s = fabs(ri) / V;
            v[1] = (s != s || v[1] != v[1]) ? NAN : fmax(v[1], s);
            v[2] = fmax(v[2], aacc / V);
            v[3] = fmax(v[3], fabs(bi) / V);
        }
    }
    publish_fold<5>(v, 0xEu, partial, counter, [&](const double (&t)[5]) {
        if (First) after_first(t, q, S, c);
        else after_run(t, q, S, c);
    });
}

// k_pres on a constant-coefficient 16x16 finest level (vectorized quads,
// stencil4.cuh): the row is c0 (count x_c - sum of neighbours), evaluated as
// c0 sum (x_c - x_nb) like k_pres; |A| |x| = |c0| (count |x_c| + sum |neighbours|).
// Every array is 16-byte aligned but the caller's solution, which `wide` says.
template <bool First>
__global__ void __launch_bounds__(256) v_pres(SView<double> L, PresIo io, int wide, SolveAsk q, double* partial,
                                              unsigned* counter, SolveState* S, CgState* c) {
    pdl_entry();
    const double mx = First ? S->mx : S->xm, mb = First ? S->mb : 0.0;
    const bool store = First || S->ok;
    double v[5] = {0, 0, 0, 0, 0};
    const int groups = (L.nblocks + 3) / 4;
    const double* vol = L.vol;
    const double ac0 = fabs(L.c0);
    for (int grp = blockIdx.x; grp < groups; grp += gridDim.x) {
        const QPos p = q_pos(grp);
        const bool valid = p.b < L.nblocks;
        // a level of equal positive volumes needs no per-cell volume loads
        const bool uniform = L.const_vol && L.vol0 > 0;
        const QNb<double> g = q_gather<double>(
            L, p, valid, [&](int k) { return q_ldv(io.xin + k); },
            [&](double xv, int k) { return (uniform || vol[k] > 0) ? xv - mx : 0.0; });
        if (!valid) continue;
        const Quad<double> vq = uniform ? Quad<double>{{L.vol0, L.vol0, L.vol0, L.vol0}} : q_ld(vol + p.c);
        Quad<double> bq = q_ldv((First ? io.rhs : io.b) + p.c), rq;
        for (int m = 0; m < 4; ++m) {
            const bool hw = m > 0 || g.hw, he = m < 3 || g.he;
            const double xc = g.x.v[m];
            double nb = 0.0, diff = 0.0;
            int cnt = 0;
            if (hw) {
                const double t = m > 0 ? g.x.v[m - 1] : g.w;
                nb += fabs(t), diff += xc - t, ++cnt;
            }
            if (he) {
                const double t = m < 3 ? g.x.v[m + 1] : g.e;
                nb += fabs(t), diff += xc - t, ++cnt;
            }
            if (g.hs) nb += fabs(g.s.v[m]), diff += xc - g.s.v[m], ++cnt;
            if (g.hn) nb += fabs(g.n.v[m]), diff += xc - g.n.v[m], ++cnt;
            const double aacc = ac0 * (double(cnt) * fabs(xc) + nb);
            const double axm = L.c0 * diff;
            const double V = vq.v[m];
            double bi = bq.v[m];
            if (First) {
                bi = V > 0 ? bi * V : 0.0;
                if (mb != 0.0 && V > 0) bi -= V * mb;
                bq.v[m] = bi;
            }
            const double ri = bi - axm;
            rq.v[m] = ri;
            v[4] += ri;
            if (V > 0) {
                v[0] += ri * ri / V;
                const double s = fabs(ri) / V;
                v[1] = (s != s || v[1] != v[1]) ? NAN : fmax(v[1], s);
                v[2] = fmax(v[2], aacc / V);
                v[3] = fmax(v[3], fabs(bi) / V);
            }
        }
        if (First) q_st(io.b + p.c, bq);
        if (store) {
            if (wide) q_st(io.xout + p.c, g.x);
            else
                for (int m = 0; m < 4; ++m) io.xout[p.c + m] = g.x.v[m];
        }
        q_st(io.r + p.c, rq);
    }
    publish_fold<5>(v, 0xEu, partial, counter, [&](const double (&t)[5]) {
        if (First) after_first(t, q, S, c);
        else after_run(t, q, S, c);
    });
}

// the iterate's mean sum V x / cvol, taken off by the next residual pass (none
// when no run was made).  vol null: every cell's volume is vol0.
__global__ void k_xmean(int n, const double* x, const double* __restrict__ vol, double vol0, double cvol,
                        double* partial, unsigned* counter, SolveState* S) {
    pdl_entry();
    double v[1] = {0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v[0] += (vol ? vol[i] : vol0) * x[i];
    publish_fold<1>(v, 0u, partial, counter, [&](const double (&t)[1]) { S->xm = S->skip ? 0.0 : t[0] / cvol; });
}

}  // namespace

void DeviceSolver::solve_fast(const double* rhs, double* x_user, double rtol, double atol, int max_cycles,
                              int compatibility, int precision, SolveStats& st) {
    DevLevel& L = levels_[0];
    const int n = L.n;
    const LevelView<double>& A = vd_[0];
    // programmatic launch only behind a kernel of this solve (not behind the
    // caller's work or a graph)
    const Launch go{stream_, pdl_}, plain{stream_, false};
    const int64_t want = (int64_t(n) + kThreads - 1) / kThreads;
    const double* vol = L.const_vol ? nullptr : A.vol;
    SolveState* S = reinterpret_cast<SolveState*>(sstate_.p);
    CgState* cg = reinterpret_cast<CgState*>(cgs_.p);
    const SolveState& hs = *host_solve_;
    SolveAsk ask;
    ask.rtol = rtol;
    ask.atol = atol;
    ask.cvol = L.ncomp == 1 ? L.comp_volume[0] : 0.0;
    // precision 2, FP64 iterative refinement: each run is a CG on the correction
    // with FP32 r, directions and Ap (x and every inner product stay FP64),
    // started from the FP32 rounding of the true residual and stopped at a fixed
    // reduction of it or at the target; its recurrence residual follows the true
    // one to about the FP32 unit roundoff per iteration
    ask.eta = precision == 2 ? ir_eta_ : 0.0;
    ask.max_cycles = max_cycles;
    ask.strict = compatibility == 1 ? 1 : 0;
    double vt = 0;  // total volume of cells with V > 0
    for (double v : L.comp_volume) vt += v;
    if (L.ncomp == 0) vt = vol_total_;
    // the refinement's runs need the multi-launch cycle
    const bool no_run = precision == 2 && coop_grid_ > 0;
    if (precision == 2 && !no_run) ensure_ir();
    TPA_CUDA(cudaEventRecord(ev0_, stream_));
    st = SolveStats();

    plain(k_prep, fold_grid(k_prep, kThreads, want, kGrid), kThreads, 0, n, rhs, (const double*)x_user, vol, L.vol0, ask,
       spartial_.p, counters_.p + kCPrep, S);
    auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    const bool vec = sdev_[0].vec;
    PresIo first{rhs, x_user, b_.p, xw_.p, r_.p};
    if (vec && !(aligned(rhs) && aligned(x_user))) {
        // the vectorized pass reads 16 bytes at a time
        TPA_CUDA(cudaMemcpyAsync(b_.p, rhs, sizeof(double) * size_t(n), cudaMemcpyDeviceToDevice, stream_));
        TPA_CUDA(cudaMemcpyAsync(tmp_.p, x_user, sizeof(double) * size_t(n), cudaMemcpyDeviceToDevice, stream_));
        first.rhs = b_.p;
        first.xin = tmp_.p;
    }
    auto pres = [&](auto is_first, const PresIo& io, const Launch& launch) {
        constexpr bool F = decltype(is_first)::value;
        if (vec)
            launch(v_pres<F>, fold_grid(v_pres<F>, 256, (sd_[0].nblocks + 3) / 4, kGrid), 256, 0, sd_[0], io,
               aligned(io.xout) ? 1 : 0, ask, spartial_.p, counters_.p + kCPres, S, cg);
        else
            launch(k_pres<F>, fold_grid(k_pres<F>, kThreads, want, kGrid), kThreads, 0, A, io, L.any_void ? 1 : 0, ask,
               spartial_.p, counters_.p + kCPres, S, cg);
    };
    pres(std::true_type(), first, first.rhs == rhs ? go : plain);
    launches_ += 2;
    if (no_run && max_cycles > 0) {
        // refused where a run is due, with the caller's solution untouched
        TPA_CUDA(cudaMemcpyAsync(host_solve_, S, sizeof(SolveState), cudaMemcpyDeviceToHost, stream_));
        TPA_CUDA(cudaStreamSynchronize(stream_));
        if (!hs.skip) ensure_ir();
    }
    double target = 0, init_linf = 0;
    auto guarded = [&](double cur, double fl) {
        if (!(std::isfinite(init_linf) && std::isfinite(cur) && target < cur && cur < init_linf)) return target;
        return (std::isfinite(fl) && fl < init_linf / 100) ? std::max(target, fl) : target;
    };
    for (bool first_run = true;; first_run = false) {
        if (max_cycles > 0 && !no_run) cg_loop(precision);
        // a run whose cooperative cycle gave up ends here, before the caller's
        // solution is written
        if (coop_grid_ > 0) check_barrier();
        // gauge of the iterate, then the true residual and its norms
        if (L.ncomp == 1) {
            plain(k_xmean, fold_grid(k_xmean, kThreads, want, kGrid), kThreads, 0, n, (const double*)xw_.p, vol, L.vol0,
               ask.cvol, spartial_.p, counters_.p + kCMean, S);
            ++launches_;
        }
        pres(std::false_type(), PresIo{nullptr, xw_.p, b_.p, x_user, r_.p}, L.ncomp == 1 ? go : plain);
        ++launches_;
        TPA_CUDA(cudaMemcpyAsync(host_solve_, S, sizeof(SolveState), cudaMemcpyDeviceToHost, stream_));
        TPA_CUDA(cudaEventRecord(ev1_, stream_));
        TPA_CUDA(cudaStreamSynchronize(stream_));
        TPA_CUDA(cudaGetLastError());
        if (first_run) {
            if (!std::isfinite(hs.abs_b)) throw Error(4, "right-hand side must be finite");
            if (!hs.ok) throw Error(1, "Poisson right-hand side has nonzero volume mean");
            target = hs.target;
            init_linf = hs.init[1];
            if (hs.skip) break;
        }
        count_cg_bodies(precision, hs.niter, hs.flags);
        ++st.restarts;
        const double linf = hs.fin[1];
        if (linf <= guarded(linf, roundoff_floor(hs.fin[2], hs.fin[3]))) break;
        if (!std::isfinite(linf) || hs.niter == 0 || hs.total >= max_cycles) break;
    }
    auto l2 = [&](double s) { return vt > 0 ? std::sqrt(s / vt) : 0.0; };
    const double tfinal = guarded(hs.fin[1], roundoff_floor(hs.fin[2], hs.fin[3]));
    float ms = 0;
    cudaEventElapsedTime(&ms, ev0_, ev1_);
    if (L.ncomp == 1) {
        st.removed_rhs_mean = hs.mb;
        st.removed_max_component_mean = std::fabs(hs.mb);
    }
    st.cycles = hs.total;
    st.converged = std::isfinite(hs.fin[1]) && std::isfinite(tfinal) && hs.fin[1] <= tfinal;
    st.initial_l2 = l2(hs.init[0]);
    st.initial_linf = hs.init[1];
    st.final_l2 = l2(hs.fin[0]);
    st.final_linf = hs.fin[1];
    st.target_linf = tfinal;
    st.residual_scale = std::max(hs.init[1], kEps);
    st.ms_total = ms;
}

}  // namespace tpa
