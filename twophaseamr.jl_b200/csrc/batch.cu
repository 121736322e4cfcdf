// Merged batch of independent pressure solves (batch.cuh): host assembly of
// the batch levels from the problems' hierarchies, the per-problem FP64 CG
// kernels, and the solve driver (one graph launch per Krylov run of the whole
// batch).  Each problem follows `solve!` (src/solvers/multigrid/
// elliptic_solver.jl:628-675 of ronaldremmerswaal/TwoPhaseAMR.jl): b = V f,
// component projection, CG with the strong-residual callback, restarts from the
// true residual (`_run_krylov_reliably!`, :487-526) and the final gauge.
#include "batch.hpp"

#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "launch.cuh"

namespace tpa {
namespace {

// ---- fine-space FP64 kernels (one BFItem per CTA) --------------------------------

// the slice of this thread's q-th row (row q kItemRows + threadIdx.x of item blockIdx.x)
__device__ __forceinline__ int2 fine_slice(const FineRows& A, int q) {
    return ld_static(A.slice + size_t(blockIdx.x) * (kFineRows / 32) + size_t(q) * (kItemRows / 32) +
                     (threadIdx.x >> 5));
}

__device__ __forceinline__ BFItem fine_item(const BFItem* fi) {
    const int* p = reinterpret_cast<const int*>(fi + blockIdx.x);
    return BFItem{ld_static(p), ld_static(p + 1), ld_static(p + 2), ld_static(p + 3), ld_static(p + 4)};
}

template <int N, typename F>
__device__ __forceinline__ void fine_fold(const FineFold& f, const double (&v)[N], unsigned max_mask, int prob,
                                          F done) {
    fold_problem<N>(v, max_mask, f.partial, f.stride, f.counters + prob, f.first[prob], f.count[prob], done);
}

// Per problem: sums of b = V f, |b| and V x0, the means to remove, and whether
// the right-hand side is accepted (compatibility = :error).
__global__ void bk_prep(const BFItem* fi, FineFold f, const double* __restrict__ vol, const double* __restrict__ rhs,
                        const double* __restrict__ xin, const double* __restrict__ comp_vol, SolveAsk q,
                        SolveState* S) {
    const BFItem it = fine_item(fi);
    double v[3] = {0, 0, 0};
#pragma unroll
    for (int q4 = 0; q4 < kFinePer; ++q4) {
        const int i = it.begin + q4 * kItemRows + int(threadIdx.x);
        if (i >= it.end) continue;
        const double V = vol[i];
        const double bi = V > 0 ? rhs[i] * V : 0.0, xi = V > 0 ? xin[i] : 0.0;
        v[0] += bi;
        v[1] += fabs(bi);
        v[2] += V * xi;
    }
    fine_fold<3>(f, v, 0u, it.prob, [&](const double (&t)[3]) {
        SolveState& s = S[it.prob];
        const double cv = comp_vol[it.prob];
        s.abs_b = t[1];
        s.ok = !(q.strict && cv > 0 && fabs(t[0]) > 256 * kEps * std_max(1.0, t[1]));
        s.mb = cv > 0 && s.ok ? t[0] / cv : 0.0;
        s.mx = cv > 0 ? t[2] / cv : 0.0;
        s.xm = 0;
    });
}

// Per problem: r = b - A x with the norms and the roundoff floor's inputs, as
// k_pres of the single solve.  First: b = V f - V mb and x = x_in - mx are formed
// and stored, the targets set and the problems that have something to solve
// started; else x - xm goes to the caller's array and the run is accounted.
// A x is summed as sum_j a_ij (x_j - x_i): the rows sum to zero, and this form
// rounds at the level of the face fluxes, as the factorized action does, rather
// than at that of a_ii x_i.
template <bool First>
__global__ void bk_pres(const BFItem* fi, FineFold f, FineRows A, const double* rhs, const double* xin, double* b,
                        double* xout, double* r, SolveAsk q, SolveState* S, BState* st, int* active) {
    const BFItem it = fine_item(fi);
    const SolveState& s = S[it.prob];
    const double m = First ? s.mx : s.xm, mb = First ? s.mb : 0.0;
    double v[5] = {0, 0, 0, 0, 0};
    for (int q4 = 0; q4 < kFinePer; ++q4) {
        const int i = it.begin + q4 * kItemRows + int(threadIdx.x);
        if (i >= it.end) continue;
        const int2 sl = fine_slice(A, q4);
        const double V = A.vol[i];
        double bi;
        if (First) {
            bi = V > 0 ? rhs[i] * V : 0.0;
            if (mb != 0.0) bi -= V * mb;
            b[i] = bi;
        } else {
            bi = b[i];
        }
        const double xi = First && !(V > 0) ? -m : xin[i] - m;
        double acc = 0, aacc = 0;
        const int* ci = A.ci + 32 * size_t(sl.x) + (threadIdx.x & 31);
        const double* val = A.val + 32 * size_t(sl.x) + (threadIdx.x & 31);
#pragma unroll 4
        for (int u = 0; u < sl.y; ++u) {
            const int j = ci[32 * u];
            const double a = val[32 * u];
            const double xj = First && !(A.vol[j] > 0) ? -m : xin[j] - m;
            acc += a * (xj - xi);
            aacc += fabs(a) * fabs(xj);
        }
        xout[i] = xi;
        const double ri = bi - acc;
        r[i] = ri;
        v[4] += ri;
        if (V > 0) {
            v[0] += ri * ri / V;
            v[1] = nan_max(v[1], fabs(ri) / V);
            v[2] = nan_max(v[2], aacc / V);
            v[3] = nan_max(v[3], fabs(bi) / V);
        }
    }
    fine_fold<5>(f, v, 0xEu, it.prob, [&](const double (&t)[5]) {
        SolveState& z = S[it.prob];
        if (First) {
            after_first(t, q, &z, st + it.prob);
            active[it.prob] = z.skip ? 0 : 1;
        } else if (!z.skip) {
            after_run(t, q, &z, st + it.prob);
        } else {
            for (int k = 0; k < 4; ++k) z.fin[k] = t[k];
        }
    });
}

// the iterate's mean per problem, taken off by the next residual pass
__global__ void bk_xmean(const BFItem* fi, FineFold f, const double* __restrict__ vol, const double* x,
                         const double* __restrict__ comp_vol, SolveState* S) {
    const BFItem it = fine_item(fi);
    double v[1] = {0};
#pragma unroll
    for (int q4 = 0; q4 < kFinePer; ++q4) {
        const int i = it.begin + q4 * kItemRows + int(threadIdx.x);
        if (i < it.end) v[0] += vol[i] * x[i];
    }
    fine_fold<1>(f, v, 0u, it.prob, [&](const double (&t)[1]) {
        const double cv = comp_vol[it.prob];
        S[it.prob].xm = cv > 0 && S[it.prob].ok ? t[0] / cv : 0.0;
    });
}

// problems that run again (their states were prepared by the last residual pass)
__global__ void bk_restart(int count, const int* again, SolveState* S, int* active) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    S[k].skip = again[k] ? 0 : 1;
    active[k] = again[k];
}

__device__ __forceinline__ void balpha(double pAp, BState* s) {
    s->pAp = pAp;
    if (pAp <= kEps * s->pnorm2 && fabs(pAp) <= kEps * s->pnorm2) {
        s->flags |= 2;
        s->alpha = 0;
    } else {
        s->alpha = s->gamma / pAp;
    }
}

// Ap = A p and alpha; the first row's entries (up to 8) in flight before the wait
__global__ void __launch_bounds__(kItemRows)
    bk_cg_ap(const BFItem* fi, FineFold f, FineRows A, const double* p, double* ap, BState* st, const int* active) {
    pdl_launch();
    const BFItem it = fine_item(fi);
    constexpr int kPre = 8;
    int c[kPre];
    double a[kPre];
    int2 sl;
    auto load = [&](int q) {
        sl = fine_slice(A, q);
        const size_t at = 32 * size_t(unsigned(sl.x)) + (threadIdx.x & 31);
#pragma unroll
        for (int u = 0; u < kPre; ++u)
            if (u < sl.y) {
                c[u] = ld_static(A.ci + at + 32 * u);
                a[u] = ld_static(A.val + at + 32 * u);
            }
    };
    load(0);
    pdl_wait();
    if (!active[it.prob]) return;
    double v[1] = {0};
    for (int q = 0; q < kFinePer; ++q) {
        const int i = it.begin + q * kItemRows + int(threadIdx.x);
        if (q) load(q);
        if (i >= it.end) continue;
        double y = 0;
#pragma unroll
        for (int u = 0; u < kPre; ++u)
            if (u < sl.y) y += a[u] * p[c[u]];
        for (int u = kPre; u < sl.y; ++u) {
            const size_t at = 32 * size_t(unsigned(sl.x)) + size_t(32 * u) + (threadIdx.x & 31);
            y += A.val[at] * p[A.ci[at]];
        }
        ap[i] = y;
        v[0] += p[i] * y;
    }
    fine_fold<1>(f, v, 0u, it.prob, [&](const double (&t)[1]) { balpha(t[0], st + it.prob); });
}

__global__ void __launch_bounds__(kItemRows)
    bk_cg_update(const BFItem* fi, FineFold f, const double* __restrict__ vol, double* x, double* r, const double* p,
                 const double* ap, BState* st, const int* active) {
    pdl_launch();
    const BFItem it = fine_item(fi);
    double V[kFinePer];
#pragma unroll
    for (int q = 0; q < kFinePer; ++q) {
        const int i = it.begin + q * kItemRows + int(threadIdx.x);
        V[q] = i < it.end ? ld_static(vol + i) : 0.0;
    }
    pdl_wait();
    if (!active[it.prob]) return;
    const bool skip = st[it.prob].flags & 2;
    const double alpha = st[it.prob].alpha;
    double ri[kFinePer], xi[kFinePer], pi[kFinePer], ai[kFinePer];
#pragma unroll
    for (int q = 0; q < kFinePer; ++q) {
        const int i = it.begin + q * kItemRows + int(threadIdx.x);
        if (i >= it.end) continue;
        ri[q] = r[i];
        xi[q] = x[i];
        pi[q] = p[i];
        ai[q] = ap[i];
    }
    double v[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < kFinePer; ++q) {
        const int i = it.begin + q * kItemRows + int(threadIdx.x);
        if (i >= it.end) continue;
        if (!skip) {
            x[i] = xi[q] + alpha * pi[q];
            ri[q] -= alpha * ai[q];
            r[i] = ri[q];
        }
        if (V[q] > 0) v[0] = nan_max(v[0], fabs(ri[q]) / V[q]);
        v[1] += ri[q];
    }
    fine_fold<2>(f, v, 1u, it.prob, [&](const double (&t)[2]) {
        st[it.prob].strong_max = t[0];
        st[it.prob].rsum = t[1];
    });
}

// p = z + beta p, z = V-cycle output - mean (not stored); a run's first: p = z
template <typename T>
__global__ void __launch_bounds__(kItemRows)
    bk_cg_p(const BFItem* fi, const BLevel<T>* __restrict__ lv, const double* mean, double* p, const BState* st,
            const int* active) {
    pdl_launch();
    const BFItem it = fine_item(fi);
    const T* xv = lv[it.lvl].x;
    pdl_wait();
    if (!active[it.prob]) return;
    const BState& s = st[it.prob];
    if (s.flags & 6) return;
    const double m = mean[it.prob], beta = s.beta;
    const bool fresh = s.iter == 0;
#pragma unroll
    for (int q = 0; q < kFinePer; ++q) {
        const int i = it.begin + q * kItemRows + int(threadIdx.x);
        if (i >= it.end) continue;
        const double z = double(xv[i + it.off]) - m;
        p[i] = fresh ? z : z + beta * p[i];
    }
}

// loop condition of the graph: any problem still iterating
__global__ void bk_cg_cond(const int* active, int count, cudaGraphConditionalHandle handle) {
    pdl_entry();
    __shared__ int any;
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < count; k += blockDim.x)
        if (active[k]) any = 1;
    __syncthreads();
    if (threadIdx.x == 0) cudaGraphSetConditional(handle, any ? 1u : 0u);
}

template <typename T>
std::vector<T> cast_vec(const std::vector<double>& v) {
    return std::vector<T>(v.begin(), v.end());
}

}  // namespace

// ---------------------------------------------------------------------------------

BatchSolver::BatchSolver(int device, const std::vector<const Hierarchy*>& hs) : device_(device) {
    TPA_CUDA(cudaSetDevice(device_));
    TPA_CUDA(cudaStreamCreateWithFlags(&own_stream_, cudaStreamNonBlocking));
    stream_ = own_stream_;
    TPA_CUDA(cudaEventCreateWithFlags(&ev_order_, cudaEventDisableTiming));
    build(hs);
}

BatchSolver::~BatchSolver() {
    cudaSetDevice(device_);
    for (auto& e : exec_)
        if (e) cudaGraphExecDestroy(e);
    if (host_state_) cudaFreeHost(host_state_);
    if (ev0_) cudaEventDestroy(ev0_);
    if (ev1_) cudaEventDestroy(ev1_);
    if (ev_order_) cudaEventDestroy(ev_order_);
    if (own_stream_) cudaStreamDestroy(own_stream_);
}

void BatchSolver::build(const std::vector<const Hierarchy*>& hs) {
    const int K = int(hs.size());
    if (K <= 0) throw Error(1, "a batch needs at least one problem");
    K_ = K;
    int Lmax = 0;
    for (const Hierarchy* h : hs) {
        if (!h || h->levels.empty()) throw Error(7, "every problem needs a hierarchy");
        if (h->levels.size() < 2) throw Error(5, "the batched solve needs at least two levels per problem");
        if (h->coarse_n != h->levels.back().op.A.n ||
            h->coarse_inverse.size() != size_t(h->coarse_n) * size_t(h->coarse_n))
            throw Error(7, "coarsest-level inverse does not match the coarsest level");
        if (h->opts.pre_sweeps != 2 || h->opts.post_sweeps != 2)
            throw Error(5, "the batched solve runs the default cycle (two pre- and two post-sweeps)");
        for (const HostLevel& l : h->levels)
            if (l.op.singular && l.op.comp.volume.size() > 1)
                throw Error(5, "the batched solve supports one ungauged component per level");
        Lmax = std::max(Lmax, int(h->levels.size()));
    }
    L_ = Lmax;
    // row offsets per level and problem
    std::vector<std::vector<int64_t>> M(size_t(Lmax), std::vector<int64_t>(size_t(K), -1));
    std::vector<int64_t> nlev(size_t(Lmax), 0);
    for (int j = 0; j < Lmax; ++j)
        for (int k = 0; k < K; ++k) {
            const int Lk = int(hs[size_t(k)]->levels.size());
            const int l = j - (Lmax - Lk);
            if (l < 0) continue;
            M[size_t(j)][size_t(k)] = nlev[size_t(j)];
            nlev[size_t(j)] += hs[size_t(k)]->levels[size_t(l)].op.A.n;
        }
    for (int64_t n : nlev)
        if (n >= (int64_t(1) << 31) - kItemRows) throw Error(5, "batch level too large for 32-bit rows");
    // fine space (problem order)
    F_.assign(size_t(K) + 1, 0);
    for (int k = 0; k < K; ++k) F_[size_t(k) + 1] = F_[size_t(k)] + hs[size_t(k)]->levels[0].op.A.n;
    if (F_[size_t(K)] >= (int64_t(1) << 31) - kItemRows) throw Error(5, "batch too large for 32-bit rows");
    nfine_ = F_[size_t(K)];

    auto level_of = [&](int j, int k) -> const HostLevel& {
        const Hierarchy& h = *hs[size_t(k)];
        return h.levels[size_t(j - (Lmax - int(h.levels.size())))];
    };
    // how a level runs: on tiles (csrc/tiles.hpp) when it is small enough and every
    // problem's share can be tiled, else streamed
    int tiles_max = kBatchTiles;
    if (const char* e = std::getenv("TPAGMG_BATCH_TILES")) tiles_max = std::max(0, std::atoi(e));
    std::vector<std::vector<TileLevelHost>> tl(static_cast<size_t>(Lmax));
    std::vector<char> on_tiles(size_t(Lmax), 0);
    std::vector<std::pair<int, int>> pairs;  // (batch level, problem) of the candidates
    for (int j = 0; j + 1 < Lmax; ++j) {
        int64_t blocks = 0;
        for (int k = 0; k < K; ++k)
            if (M[size_t(j)][size_t(k)] >= 0) blocks += level_of(j, k).op.mesh.nblocks();
        on_tiles[size_t(j)] = blocks <= tiles_max;
        if (!on_tiles[size_t(j)]) continue;
        tl[size_t(j)].resize(size_t(K));
        for (int k = 0; k < K; ++k)
            if (M[size_t(j)][size_t(k)] >= 0) pairs.emplace_back(j, k);
    }
#pragma omp parallel for schedule(dynamic, 1)
    for (size_t q = 0; q < pairs.size(); ++q) {
        const int j = pairs[q].first, k = pairs[q].second;
        try {
            const HostLevel& hl = level_of(j, k);
            const Mesh& m = hl.op.mesh;
            tl[size_t(j)][size_t(k)] = build_tiles(hl.op.A, m.nblocks(), m.cells_per_block(), hl.owner,
                                                   level_of(j + 1, k).op.A.n, kTileMaxCells);
        } catch (...) {
            tl[size_t(j)][size_t(k)].ok = false;
        }
    }
    for (const auto& q : pairs)
        if (!tl[size_t(q.first)][size_t(q.second)].ok) on_tiles[size_t(q.first)] = 0;

    lev_.clear();
    lev_.resize(size_t(Lmax));
    btl_.clear();
    btl_.resize(size_t(Lmax));
    int64_t max_items = 0;
    for (int j = 0; j < Lmax; ++j) {
        BLevelHost& H = lev_[size_t(j)];
        H.n = int(nlev[size_t(j)]);
        std::vector<double> wd(size_t(H.n)), td(size_t(H.n)), vol(size_t(H.n)), cvol(size_t(K), 0.0);
        std::vector<int64_t> delta(size_t(K), kNoExt);
        std::vector<const HostLevel*> hl(size_t(K), nullptr);
        for (int k = 0; k < K; ++k) {
            if (M[size_t(j)][size_t(k)] < 0) continue;
            hl[size_t(k)] = &level_of(j, k);
            if (hl[size_t(k)] == &hs[size_t(k)]->levels[0]) delta[size_t(k)] = F_[size_t(k)] - M[size_t(j)][size_t(k)];
        }
#pragma omp parallel for schedule(dynamic, 1)
        for (int k = 0; k < K; ++k) {
            if (!hl[size_t(k)]) continue;
            const HostLevel& h = *hl[size_t(k)];
            const size_t off = size_t(M[size_t(j)][size_t(k)]);
            for (size_t i = 0; i < size_t(h.op.A.n); ++i) {
                wd[off + i] = h.weight * h.inv_diag[i];
                td[off + i] = h.transfer_inv.empty() ? 0.0 : h.transfer_weight * h.transfer_inv[i];
                vol[off + i] = h.op.volumes[i];
            }
            if (h.op.singular && !h.op.comp.volume.empty()) cvol[size_t(k)] = 1.0 / h.op.comp.volume[0];
        }
        if (j + 1 < Lmax) {
            if (on_tiles[size_t(j)])
                merge_tiles(btl_[size_t(j)], H, tl[size_t(j)], hl, M[size_t(j)], M[size_t(j) + 1], delta);
            else
                merge_rows(H, hl, M[size_t(j)], M[size_t(j) + 1], delta);
            tl[size_t(j)].clear();
            max_items = std::max<int64_t>(max_items, std::max(H.nitems, btl_[size_t(j)].ntiles));
        }
        H.cvol_inv.upload(cvol.data(), cvol.size(), stream_);
        H.wd_d.upload(wd.data(), wd.size(), stream_);
        H.td_d.upload(td.data(), td.size(), stream_);
        H.vol_d.upload(vol.data(), vol.size(), stream_);
        {
            auto g = cast_vec<float>(wd);
            H.wd_f.upload(g.data(), g.size(), stream_);
            auto t = cast_vec<float>(td);
            H.td_f.upload(t.data(), t.size(), stream_);
            auto v = cast_vec<float>(vol);
            H.vol_f.upload(v.data(), v.size(), stream_);
            TPA_CUDA(cudaStreamSynchronize(stream_));
        }
        for (auto* a : {&H.b_d, &H.bp_d, &H.x_d, &H.y_d}) a->alloc(size_t(H.n));
        for (auto* a : {&H.b_f, &H.bp_f, &H.x_f, &H.y_f}) a->alloc(size_t(H.n));
        if (H.nitems) {
            H.r_d.alloc(size_t(H.n));
            H.r_f.alloc(size_t(H.n));
        }
        TPA_CUDA(cudaStreamSynchronize(stream_));
    }
    // views
    vd_.assign(size_t(Lmax), BLevel<double>{});
    vf_.assign(size_t(Lmax), BLevel<float>{});
    for (int j = 0; j < Lmax; ++j) {
        BLevelHost& H = lev_[size_t(j)];
        auto fill = [&](auto& v, auto& val, auto& wd, auto& td, auto& vol, auto& b, auto& bp, auto& x, auto& y,
                        auto& r) {
            v.wd = wd.p;
            v.td = td.p;
            v.vol = vol.p;
            v.cvol_inv = H.cvol_inv.p;
            v.b = b.p;
            v.bp = bp.p;
            v.x = x.p;
            v.y = y.p;
            v.r = r.p;
            v.items = H.items.p;
            v.slice = reinterpret_cast<const int2*>(H.slice.p);
            v.val = val.p;
            v.ci = H.ci.p;
            v.cc = H.cc.p;
            v.owner = H.owner.p;
            v.cptr = H.cptr.p;
            v.co = H.co.p;
            v.ch = reinterpret_cast<const short4*>(H.ch.p);
            v.pfirst = H.pfirst.p;
            v.pcount = H.pcount.p;
            v.sprob = H.sprob.p;
            v.sch = reinterpret_cast<const int4*>(H.sch.p);
            v.nsplit = H.nsplit;
            v.nitems = H.nitems;
        };
        fill(vd_[size_t(j)], H.val_d, H.wd_d, H.td_d, H.vol_d, H.b_d, H.bp_d, H.x_d, H.y_d, H.r_d);
        fill(vf_[size_t(j)], H.val_f, H.wd_f, H.td_f, H.vol_f, H.b_f, H.bp_f, H.x_f, H.y_f, H.r_f);
    }
    vd_dev_.upload(vd_.data(), vd_.size(), stream_);
    vf_dev_.upload(vf_.data(), vf_.size(), stream_);
    // tails and coarse inverses
    {
        std::vector<double> G;
        std::vector<int64_t> goff(static_cast<size_t>(K));
        for (int k = 0; k < K; ++k) {
            goff[size_t(k)] = int64_t(G.size());
            G.insert(G.end(), hs[size_t(k)]->coarse_inverse.begin(), hs[size_t(k)]->coarse_inverse.end());
        }
        G_.upload(G.data(), G.size(), stream_);
        TPA_CUDA(cudaStreamSynchronize(stream_));
        std::vector<BCoarse> co;
        for (int k = 0; k < K; ++k)
            for (int row = 0; row < int(hs[size_t(k)]->coarse_n); row += kCoarseRows)
                co.push_back(BCoarse{G_.p + goff[size_t(k)], int(hs[size_t(k)]->coarse_n),
                                     int(M[size_t(Lmax) - 1][size_t(k)]), row, k});
        ncoarse_ = int(co.size());
        coarse_.upload(co.data(), co.size(), stream_);
        const double ones[3] = {1.0, 1.0, 1.0};
        ones_.upload(ones, 3, stream_);
        TPA_CUDA(cudaStreamSynchronize(stream_));
    }
    // fine space: items, the FP64 rows in slices, and volumes
    {
        std::vector<BFItem> fi;
        std::vector<int> pf(static_cast<size_t>(K)), pc(static_cast<size_t>(K)), slice;
        for (int k = 0; k < K; ++k) {
            const Hierarchy& h = *hs[size_t(k)];
            const int j = Lmax - int(h.levels.size());
            const Csr& A = h.levels[0].op.A;
            const int F = int(F_[size_t(k)]);
            pf[size_t(k)] = int(fi.size());
            for (int64_t b = 0; b < A.n; b += kFineRows)
                fi.push_back(BFItem{F + int(b), F + int(std::min<int64_t>(A.n, b + kFineRows)), k, j,
                                    int(M[size_t(j)][size_t(k)]) - F});
            pc[size_t(k)] = int(fi.size()) - pf[size_t(k)];
            comp_vol_.push_back(h.levels[0].op.singular ? h.levels[0].op.comp.volume[0] : 0.0);
            double tv = 0;
            for (double v : h.levels[0].op.volumes)
                if (v > 0) tv += v;
            total_vol_.push_back(tv);
        }
        int64_t entries = 0;
        for (const BFItem& it : fi) {
            const Csr& A = hs[size_t(it.prob)]->levels[0].op.A;
            const int F = int(F_[size_t(it.prob)]);
            for (int b = 0; b < kFineRows; b += 32) {
                int width = 0;
                for (int i = it.begin + b; i < std::min(it.end, it.begin + b + 32); ++i)
                    width = std::max<int>(width, int(A.ptr[size_t(i - F) + 1] - A.ptr[size_t(i - F)]));
                if (entries / 32 > INT32_MAX - int64_t(width)) throw Error(5, "batch has too many operator entries");
                slice.push_back(int(entries / 32));
                slice.push_back(width);
                entries += 32 * int64_t(width);
            }
        }
        std::vector<int> ci(static_cast<size_t>(entries));
        std::vector<double> val(size_t(entries), 0.0), vol(static_cast<size_t>(nfine_));
#pragma omp parallel for schedule(static)
        for (size_t q = 0; q < fi.size(); ++q) {
            const BFItem& it = fi[q];
            const HostLevel& hl = hs[size_t(it.prob)]->levels[0];
            const Csr& A = hl.op.A;
            const int F = int(F_[size_t(it.prob)]);
            for (int b = 0; b < kFineRows; b += 32) {
                const size_t sl = 2 * (q * (kFineRows / 32) + size_t(b / 32));
                for (int r = 0; r < 32; ++r) {
                    const int i = it.begin + b + r;
                    const bool in = i < it.end;
                    const int64_t e0 = in ? A.ptr[size_t(i - F)] : 0, e1 = in ? A.ptr[size_t(i - F) + 1] : 0;
                    for (int u = 0; u < slice[sl + 1]; ++u) {
                        const size_t at = 32 * size_t(slice[sl]) + size_t(32 * u + r);
                        ci[at] = e0 + u < e1 ? A.col[size_t(e0 + u)] + F : (in ? i : it.begin);
                        if (e0 + u < e1) val[at] = A.val[size_t(e0 + u)];
                    }
                }
            }
            for (int i = it.begin; i < it.end; ++i) vol[size_t(i)] = hl.op.volumes[size_t(i - F)];
        }
        nfi_ = int(fi.size());
        max_items = std::max<int64_t>(max_items, nfi_);
        fitems_.upload(fi.data(), fi.size(), stream_);
        fpfirst_.upload(pf.data(), pf.size(), stream_);
        fpcount_.upload(pc.data(), pc.size(), stream_);
        fslice_.upload(slice.data(), slice.size(), stream_);
        fci_.upload(ci.data(), ci.size(), stream_);
        fval_.upload(val.data(), val.size(), stream_);
        fvol_.upload(vol.data(), vol.size(), stream_);
        fcomp_.upload(comp_vol_.data(), comp_vol_.size(), stream_);
        TPA_CUDA(cudaStreamSynchronize(stream_));
    }
    const size_t nf = size_t(nfine_);
    for (auto* a : {&b_, &x_, &r_, &p_, &ap_}) a->alloc(nf);
    stride_ = int(max_items);
    partial_.alloc(size_t(5) * size_t(max_items));
    counters_.alloc(size_t(K));
    TPA_CUDA(cudaMemsetAsync(counters_.p, 0, counters_.n * sizeof(unsigned), stream_));
    state_.alloc(size_t(K));
    sstate_.alloc(size_t(K));
    active_.alloc(size_t(K));
    again_.alloc(size_t(K));
    mean_.alloc(size_t(K));
    TPA_CUDA(cudaMemsetAsync(mean_.p, 0, size_t(K) * sizeof(double), stream_));
    TPA_CUDA(cudaMemsetAsync(state_.p, 0, size_t(K) * sizeof(BState), stream_));
    TPA_CUDA(cudaMallocHost(&host_state_, size_t(K) * sizeof(SolveState)));
    TPA_CUDA(cudaEventCreate(&ev0_));
    TPA_CUDA(cudaEventCreate(&ev1_));
    TPA_CUDA(cudaStreamSynchronize(stream_));
}

// One level's tiles over all problems: the problems' lists one after another,
// renumbered to batch-level rows.
void BatchSolver::merge_tiles(BTileHost& B, BLevelHost& H, const std::vector<TileLevelHost>& tl,
                              const std::vector<const HostLevel*>& hl, const std::vector<int64_t>& row,
                              const std::vector<int64_t>& coarse, const std::vector<int64_t>& delta) {
    const int K = K_;
    std::vector<size_t> t0(size_t(K) + 1, 0), c0(t0), s0(t0), e0(t0), o0(t0);
    std::vector<int> first(size_t(K), 0), count(size_t(K), 0);
    for (int k = 0; k < K; ++k) {
        const TileLevelHost& T = tl[size_t(k)];
        t0[size_t(k) + 1] = t0[size_t(k)] + T.info.size();
        c0[size_t(k) + 1] = c0[size_t(k)] + T.cell.size();
        s0[size_t(k) + 1] = s0[size_t(k)] + T.slice.size() / 2;
        e0[size_t(k) + 1] = e0[size_t(k)] + T.pos.size();
        o0[size_t(k) + 1] = o0[size_t(k)] + T.co.size();
        first[size_t(k)] = int(t0[size_t(k)]);
        count[size_t(k)] = int(T.info.size());
        B.n3max = std::max(B.n3max, T.n3max);
        B.n2max = std::max(B.n2max, T.n2max);
    }
    if (c0[size_t(K)] > size_t(INT32_MAX) || e0[size_t(K)] > size_t(INT32_MAX))
        throw Error(5, "batch level too large for 32-bit tile lists");
    B.ntiles = int(t0[size_t(K)]);
    B.rows = B.n2max > 1024 ? 2 : 1;
    B.nt = tile_threads(B.n3max, B.n2max, B.rows);
    std::vector<TileInfo> info(t0[size_t(K)]);
    std::vector<BTile> tiles(t0[size_t(K)]);
    std::vector<int> cell(c0[size_t(K)]), own(c0[size_t(K)]), slice(2 * s0[size_t(K)]), co(o0[size_t(K)]);
    std::vector<double> val(e0[size_t(K)]);
    std::vector<float> valf(e0[size_t(K)]);
    std::vector<int16_t> col(e0[size_t(K)]), ch(4 * o0[size_t(K)]);
#pragma omp parallel for schedule(dynamic, 1)
    for (int k = 0; k < K; ++k) {
        const TileLevelHost& T = tl[size_t(k)];
        if (T.info.empty()) continue;
        const int r = int(row[size_t(k)]), c = int(coarse[size_t(k)]);
        for (size_t q = 0; q < T.info.size(); ++q) {
            TileInfo I = T.info[q];
            I.cell += int(c0[size_t(k)]);
            I.slice += int(s0[size_t(k)]);
            I.co += int(o0[size_t(k)]);
            info[t0[size_t(k)] + q] = I;
            tiles[t0[size_t(k)] + q] = BTile{k, int(delta[size_t(k)])};
        }
        for (size_t q = 0; q < T.cell.size(); ++q) {
            cell[c0[size_t(k)] + q] = T.cell[q] + r;
            own[c0[size_t(k)] + q] = T.own[q] + c;
        }
        for (size_t q = 0; q < T.slice.size(); q += 2) {
            slice[2 * s0[size_t(k)] + q] = T.slice[q] + int(e0[size_t(k)]);
            slice[2 * s0[size_t(k)] + q + 1] = T.slice[q + 1];
        }
        const std::vector<double>& a = hl[size_t(k)]->op.A.val;
        for (size_t q = 0; q < T.pos.size(); ++q) {
            const double v = T.pos[q] >= 0 ? a[size_t(T.pos[q])] : 0.0;
            val[e0[size_t(k)] + q] = v;
            valf[e0[size_t(k)] + q] = float(v);
            col[e0[size_t(k)] + q] = T.col[q];
        }
        for (size_t q = 0; q < T.co.size(); ++q) co[o0[size_t(k)] + q] = T.co[q] + c;
        std::copy(T.ch.begin(), T.ch.end(), ch.begin() + std::ptrdiff_t(4 * o0[size_t(k)]));
    }
    B.info.upload(info.data(), info.size(), stream_);
    B.tiles.upload(tiles.data(), tiles.size(), stream_);
    H.pfirst.upload(first.data(), first.size(), stream_);
    H.pcount.upload(count.data(), count.size(), stream_);
    B.cell.upload(cell.data(), cell.size(), stream_);
    B.own.upload(own.data(), own.size(), stream_);
    B.slice.upload(slice.data(), slice.size(), stream_);
    B.co.upload(co.data(), co.size(), stream_);
    B.ch.upload(ch.data(), ch.size(), stream_);
    B.col.upload(col.data(), col.size(), stream_);
    B.val_d.upload(val.data(), val.size(), stream_);
    B.val_f.upload(valf.data(), valf.size(), stream_);
    TPA_CUDA(cudaStreamSynchronize(stream_));  // the host arrays go out of scope
}

// One level's rows over all problems, for the streamed phases: items of whole
// blocks or, of larger blocks, of whole pairs of block rows (at most kItemRows
// rows), so that the children of a coarse row lie in one item where that can be;
// the operator in slices.
void BatchSolver::merge_rows(BLevelHost& H, const std::vector<const HostLevel*>& hl, const std::vector<int64_t>& row,
                             const std::vector<int64_t>& coarse, const std::vector<int64_t>& delta) {
    const int K = K_;
    std::vector<BItem> items;
    std::vector<int> first(size_t(K), 0), count(size_t(K), 0);
    for (int k = 0; k < K; ++k) {
        first[size_t(k)] = int(items.size());
        if (!hl[size_t(k)]) continue;
        const int64_t n = hl[size_t(k)]->op.A.n, cpb = hl[size_t(k)]->op.mesh.cells_per_block();
        const int64_t unit = cpb <= kItemRows ? cpb : std::min<int64_t>(2 * hl[size_t(k)]->op.mesh.bs[0], kItemRows);
        const int64_t step = kItemRows / unit * unit;
        for (int64_t b = 0; b < n; b += step)
            items.push_back(BItem{int(row[size_t(k)] + b), int(row[size_t(k)] + std::min(n, b + step)), k,
                                  int(delta[size_t(k)])});
        count[size_t(k)] = int(items.size()) - first[size_t(k)];
    }
    const size_t ni = items.size();
    std::vector<int> slice(2 * ni * (kItemRows / 32));
    int64_t entries = 0;
    for (size_t q = 0; q < ni; ++q) {
        const Csr& A = hl[size_t(items[q].prob)]->op.A;
        const int r0 = int(row[size_t(items[q].prob)]);
        for (int w = 0; w < kItemRows / 32; ++w) {
            int64_t width = 0;
            for (int i = items[q].begin + 32 * w; i < std::min(items[q].end, items[q].begin + 32 * w + 32); ++i)
                width = std::max(width, A.ptr[size_t(i - r0) + 1] - A.ptr[size_t(i - r0)]);
            if (entries / 32 > INT32_MAX - width) throw Error(5, "batch level has too many nonzeros");
            slice[2 * (q * (kItemRows / 32) + size_t(w))] = int(entries / 32);
            slice[2 * (q * (kItemRows / 32) + size_t(w)) + 1] = int(width);
            entries += 32 * width;
        }
    }
    std::vector<int> ci(size_t(entries), 0), cc(size_t(entries), 0), own(size_t(H.n), 0), cptr(ni + 1, 0);
    std::vector<double> val(size_t(entries), 0.0);
    std::vector<float> valf(size_t(entries), 0.0f);
    std::vector<std::vector<int>> co(ni);
    std::vector<std::vector<int16_t>> ch(ni);
    int bad = 0;
#pragma omp parallel for schedule(dynamic, 16) reduction(+ : bad)
    for (size_t q = 0; q < ni; ++q) {
        const BItem& it = items[q];
        const HostLevel& h = *hl[size_t(it.prob)];
        const Csr& A = h.op.A;
        const int r0 = int(row[size_t(it.prob)]), c0 = int(coarse[size_t(it.prob)]);
        std::vector<std::pair<int, int>> kids;  // (coarse row, item-local row)
        for (int i = it.begin; i < it.end; ++i) {
            const int l = i - it.begin;
            const size_t s = 2 * (q * (kItemRows / 32) + size_t(l / 32));
            for (int u = 0; u < slice[s + 1]; ++u) {
                const size_t at = 32 * size_t(slice[s]) + size_t(32 * u + l % 32);
                const int64_t e = A.ptr[size_t(i - r0)] + u;
                const bool real = e < A.ptr[size_t(i - r0) + 1];
                const int c = real ? A.col[size_t(e)] : i - r0;
                ci[at] = c + r0;
                cc[at] = h.owner[size_t(c)] + c0;
                if (real) {
                    val[at] = A.val[size_t(e)];
                    valf[at] = float(A.val[size_t(e)]);
                }
            }
            own[size_t(i)] = h.owner[size_t(i - r0)] + c0;
            kids.emplace_back(own[size_t(i)], l);
        }
        std::stable_sort(kids.begin(), kids.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
        for (size_t a = 0; a < kids.size();) {
            int16_t q4[4] = {-1, -1, -1, -1};
            size_t b = a;
            for (; b < kids.size() && kids[b].first == kids[a].first; ++b) {
                if (b - a < 4) q4[b - a] = int16_t(kids[b].second);
                else ++bad;
            }
            co[q].push_back(kids[a].first);
            ch[q].insert(ch[q].end(), q4, q4 + 4);
            a = b;
        }
    }
    // every coarse row in exactly one item, or the rows of all items gathered
    std::vector<int> co_all;
    std::vector<int16_t> ch_all;
    for (size_t q = 0; q < ni; ++q) {
        co_all.insert(co_all.end(), co[q].begin(), co[q].end());
        ch_all.insert(ch_all.end(), ch[q].begin(), ch[q].end());
        cptr[q + 1] = int(co_all.size());
    }
    std::vector<int> once(co_all), sprob, sch;
    std::sort(once.begin(), once.end());
    if (std::adjacent_find(once.begin(), once.end()) != once.end()) {
        once.erase(std::unique(once.begin(), once.end()), once.end());
        sprob.assign(once.size(), 0);
        sch.assign(4 * once.size(), -1);
        std::vector<int> used(once.size(), 0);
        for (const BItem& it : items)
            for (int i = it.begin; i < it.end; ++i) {
                const size_t J = size_t(std::lower_bound(once.begin(), once.end(), own[size_t(i)]) - once.begin());
                sprob[J] = it.prob;
                if (used[J] < 4) sch[4 * J + size_t(used[J]++)] = i;
                else ++bad;
            }
        co_all = once;
        H.nsplit = int(once.size());
    }
    if (bad) throw Error(5, "the batched solve needs at most four children per coarse cell");
    H.sprob.upload(sprob.data(), sprob.size(), stream_);
    H.sch.upload(sch.data(), sch.size(), stream_);
    H.nitems = int(ni);
    H.items.upload(items.data(), items.size(), stream_);
    H.pfirst.upload(first.data(), first.size(), stream_);
    H.pcount.upload(count.data(), count.size(), stream_);
    H.slice.upload(slice.data(), slice.size(), stream_);
    H.ci.upload(ci.data(), ci.size(), stream_);
    H.cc.upload(cc.data(), cc.size(), stream_);
    H.owner.upload(own.data(), own.size(), stream_);
    H.cptr.upload(cptr.data(), cptr.size(), stream_);
    H.co.upload(co_all.data(), co_all.size(), stream_);
    H.ch.upload(ch_all.data(), ch_all.size(), stream_);
    H.val_d.upload(val.data(), val.size(), stream_);
    H.val_f.upload(valf.data(), valf.size(), stream_);
    TPA_CUDA(cudaStreamSynchronize(stream_));  // the host arrays go out of scope
}

// ---- one V-cycle of every active problem ------------------------------------------

// `init`: the first V-cycle of a run (its r'z starts the recurrences)
template <typename T>
void BatchSolver::enqueue_vcycle(const double* r, int init) {
    const Launch go{stream_, true};
    const std::vector<BLevel<T>>* Vp;
    if constexpr (std::is_same<T, double>::value) Vp = &vd_;
    else Vp = &vf_;
    const std::vector<BLevel<T>>& V = *Vp;
    BState* st = state_.p;
    int* act = active_.p;
    auto level = [&](int j) {
        LevelView<T> L{};
        const BLevel<T>& B = V[size_t(j)];
        L.n = lev_[size_t(j)].n;
        L.dinv = B.wd;  // the weights are folded into the rows
        L.tinv = B.td;
        L.wt = ones_.p;
        L.vol = B.vol;
        L.b = B.b;
        L.bp = B.bp;
        L.x = B.x;
        L.y = B.y;
        return L;
    };
    auto view = [&](int j) {
        const BTileHost& B = btl_[size_t(j)];
        TileView<T> W;
        W.info = B.info.p;
        W.cell = B.cell.p;
        W.own = B.own.p;
        W.slice = reinterpret_cast<const int2*>(B.slice.p);
        if constexpr (std::is_same<T, double>::value) W.val = B.val_d.p;
        else W.val = B.val_f.p;
        W.col = reinterpret_cast<const short*>(B.col.p);
        W.co = B.co.p;
        W.ch = reinterpret_cast<const short4*>(B.ch.p);
        return W;
    };
    const int last = L_ - 1;
    for (int j = 0; j < last; ++j) {
        const BTileHost& B = btl_[size_t(j)];
        const BLevel<T>& L = V[size_t(j)];
        if (L.nitems) {
            go(bk_pre2<T>, L.nitems, kItemRows, 0, L, r, (const BState*)st, (const int*)act);
            go(bk_residual<T>, L.nitems, kItemRows, 0, L, (const int*)act);
            go(bk_restrict<T>, L.nitems, kItemRows, 0, L, V[size_t(j) + 1].b, (const int*)act);
            launches_ += 3;
            if (L.nsplit) {
                go(bk_gather<T>, (L.nsplit + 255) / 256, 256, 0, L, V[size_t(j) + 1].b, (const int*)act);
                ++launches_;
            }
            continue;
        }
        const BTileRhs<T> src{B.tiles.p, L.cvol_inv, r, L.b, st, act};
        with_tile_threads(B.nt, B.rows, [&](auto nt, auto rows) {
            constexpr int NT = decltype(nt)::value, RW = decltype(rows)::value;
            go(bk_tile_down<T, NT, RW>, B.ntiles, B.nt, 0, level(j), view(j), src,
               V[size_t(j) + 1].b);
        });
        ++launches_;
    }
    go(bk_coarse<T>, ncoarse_, 32 * kCoarseRows, 0, (const BCoarse*)coarse_.p, (const T*)V[size_t(last)].b,
       V[size_t(last)].x, (const int*)act);
    ++launches_;
    for (int j = last - 1; j >= 0; --j) {
        const BTileHost& B = btl_[size_t(j)];
        const BLevel<T>& L = V[size_t(j)];
        const T* xc = V[size_t(j) + 1].x;
        if (L.nitems) {
            go(bk_prolong<T>, L.nitems, kItemRows, 0, L, xc, (const int*)act);
            go(bk_post<T, false>, L.nitems, kItemRows, 0, L, (const T*)L.x, L.y, r, partial_.p, stride_, counters_.p,
               mean_.p, st, act, init);
            go(bk_post<T, true>, L.nitems, kItemRows, 0, L, (const T*)L.y, L.x, r, partial_.p, stride_, counters_.p,
               mean_.p, st, act, init);
            launches_ += 3;
            continue;
        }
        with_tile_threads(B.nt, B.rows, [&](auto nt, auto rows) {
            constexpr int NT = decltype(nt)::value, RW = decltype(rows)::value;
            go(bk_tile_up<T, NT, RW>, B.ntiles, B.nt, 0, level(j), view(j),
               (const BTile*)B.tiles.p, L.cvol_inv, xc, r, L.pfirst, L.pcount, partial_.p, stride_, counters_.p,
               mean_.p, st, act, init);
        });
        ++launches_;
    }
}

FineFold BatchSolver::fine_fold_args() const {
    return FineFold{fpfirst_.p, fpcount_.p, partial_.p, stride_, counters_.p};
}

FineRows BatchSolver::fine_rows() const {
    return FineRows{reinterpret_cast<const int2*>(fslice_.p), fci_.p, fval_.p, fvol_.p};
}

// z = V-cycle(r) with r'z and the stopping rules, then the direction
void BatchSolver::enqueue_direction(int precision, int init) {
    const Launch go{stream_, true};
    if (precision == 0) {
        enqueue_vcycle<double>(r_.p, init);
        go(bk_cg_p<double>, nfi_, kItemRows, 0, (const BFItem*)fitems_.p, vd_dev_.p, (const double*)mean_.p, p_.p,
           (const BState*)state_.p, (const int*)active_.p);
    } else {
        enqueue_vcycle<float>(r_.p, init);
        go(bk_cg_p<float>, nfi_, kItemRows, 0, (const BFItem*)fitems_.p, vf_dev_.p, (const double*)mean_.p, p_.p,
           (const BState*)state_.p, (const int*)active_.p);
    }
    ++launches_;
}

void BatchSolver::enqueue_body(int precision, cudaGraphConditionalHandle handle, bool in_graph) {
    const Launch go{stream_, true};
    BState* st = state_.p;
    go(bk_cg_ap, nfi_, kItemRows, 0, (const BFItem*)fitems_.p, fine_fold_args(), fine_rows(), (const double*)p_.p,
       ap_.p, st, (const int*)active_.p);
    go(bk_cg_update, nfi_, kItemRows, 0, (const BFItem*)fitems_.p, fine_fold_args(), fvol_.p, x_.p, r_.p,
       (const double*)p_.p, (const double*)ap_.p, st, (const int*)active_.p);
    launches_ += 2;
    enqueue_direction(precision, 0);
    if (in_graph) {
        go(bk_cg_cond, 1, 256, 0, (const int*)active_.p, K_, handle);
        ++launches_;
    }
}

cudaGraphExec_t BatchSolver::graph(int precision) {
    if (exec_[precision]) return exec_[precision];
    cudaGraph_t g;
    TPA_CUDA(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle handle;
    TPA_CUDA(cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault));
    alignas(cudaGraphNodeParams) unsigned char storage[sizeof(cudaGraphNodeParams)];
    std::memset(storage, 0, sizeof(storage));
    cudaGraphNodeParams& cp = *reinterpret_cast<cudaGraphNodeParams*>(storage);
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    // the loop is entered when a problem is active after its first V-cycle
    const int* act = active_.p;
    void* gate_args[] = {&act, &K_, &handle};
    cudaKernelNodeParams gate;
    std::memset(&gate, 0, sizeof(gate));
    gate.func = reinterpret_cast<void*>(bk_cg_cond);
    gate.gridDim = dim3(1);
    gate.blockDim = dim3(256);
    gate.kernelParams = gate_args;
    cudaGraphNode_t gate_node, node;
    TPA_CUDA(cudaGraphAddKernelNode(&gate_node, g, nullptr, 0, &gate));
    TPA_CUDA(cudaGraphAddNode(&node, g, &gate_node, 1, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    cudaStream_t saved = stream_;
    stream_ = own_stream_;
    const int before = launches_;
    TPA_CUDA(cudaStreamBeginCaptureToGraph(stream_, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    enqueue_body(precision, handle, true);
    cudaGraph_t captured;
    cudaError_t ce = cudaStreamEndCapture(stream_, &captured);
    stream_ = saved;
    body_launches_[precision] = launches_ - before;
    launches_ = before;
    if (ce != cudaSuccess) {
        cudaGraphDestroy(g);
        throw Error(2, std::string("batch graph capture failed: ") + cudaGetErrorString(ce));
    }
    cudaGraphExec_t exec;
    cudaError_t ie = cudaGraphInstantiate(&exec, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) throw Error(2, std::string("batch graph instantiation failed: ") + cudaGetErrorString(ie));
    exec_[precision] = exec;
    return exec;
}

// ---- the solve --------------------------------------------------------------------

void BatchSolver::solve(const double* rhs, double* x_user, double rtol, double atol, int max_cycles,
                        int compatibility, int precision, std::vector<SolveStats>& stats, std::vector<int>& status,
                        std::vector<std::string>& messages) {
    TPA_CUDA(cudaSetDevice(device_));
    if (!(rtol >= 0 && rtol < 1)) throw Error(1, "rtol must lie in [0, 1)");
    if (!(atol >= 0)) throw Error(1, "atol must be nonnegative");
    if (max_cycles < 0) throw Error(1, "max_cycles must be nonnegative");
    if (compatibility != 0 && compatibility != 1) throw Error(1, "compatibility must be :project or :error");
    if (precision != 0 && precision != 1) throw Error(1, "precision must be 0 (FP64) or 1 (mixed)");
    const int K = K_;
    const Launch plain{stream_, false};
    const FineRows A = fine_rows();
    const FineFold fold = fine_fold_args();
    BState* st = state_.p;
    SolveState* S = sstate_.p;
    const SolveState* hs = host_state_;
    SolveAsk ask;
    ask.rtol = rtol;
    ask.atol = atol;
    ask.cvol = 0;  // per problem, from fcomp_
    ask.eta = 0;
    ask.max_cycles = max_cycles;
    ask.strict = compatibility == 1 ? 1 : 0;
    stats.assign(size_t(K), SolveStats());
    status.assign(size_t(K), 0);
    messages.assign(size_t(K), std::string());
    const bool no_graph = std::getenv("TPAGMG_NO_GRAPH") != nullptr;
    TPA_CUDA(cudaEventRecord(ev0_, stream_));
    plain(bk_prep, nfi_, kItemRows, 0, (const BFItem*)fitems_.p, fold, fvol_.p, rhs, (const double*)x_user, fcomp_.p,
          ask, S);
    plain(bk_pres<true>, nfi_, kItemRows, 0, (const BFItem*)fitems_.p, fold, A, rhs, (const double*)x_user, b_.p, x_.p,
          r_.p, ask, S, st, active_.p);
    launches_ += 2;
    std::vector<int> run(size_t(K), 1), act(static_cast<size_t>(K));
    auto guarded = [&](int k, double cur) {
        const double init = hs[k].init[1], tg = hs[k].target, f = roundoff_floor(hs[k].fin[2], hs[k].fin[3]);
        if (!(std::isfinite(init) && std::isfinite(cur) && tg < cur && cur < init)) return tg;
        return (std::isfinite(f) && f < init / 100) ? std::max(tg, f) : tg;
    };
    for (bool first = true;; first = false) {
        // one Krylov run of every problem that is active
        enqueue_direction(precision, 1);
        if (no_graph) {
            // the loop body launched kernel by kernel, its condition read on the
            // host before each one (profiling and diagnosis); every problem stops
            // within its iteration limit
            const int before = launches_;
            for (int body = 0; body <= max_cycles; ++body) {
                TPA_CUDA(cudaMemcpyAsync(act.data(), active_.p, size_t(K) * sizeof(int), cudaMemcpyDeviceToHost,
                                         stream_));
                TPA_CUDA(cudaStreamSynchronize(stream_));
                if (std::none_of(act.begin(), act.end(), [](int v) { return v != 0; })) break;
                enqueue_body(precision, cudaGraphConditionalHandle(), false);
            }
            launches_ = before;  // counted from the iterations below
        } else {
            TPA_CUDA(cudaGraphLaunch(graph(precision), stream_));
        }
        plain(bk_xmean, nfi_, kItemRows, 0, (const BFItem*)fitems_.p, fold, fvol_.p, (const double*)x_.p, fcomp_.p, S);
        plain(bk_pres<false>, nfi_, kItemRows, 0, (const BFItem*)fitems_.p, fold, A, (const double*)nullptr,
              (const double*)x_.p, b_.p, x_user, r_.p, ask, S, st, active_.p);
        launches_ += 2;
        TPA_CUDA(cudaMemcpyAsync(host_state_, S, size_t(K) * sizeof(SolveState), cudaMemcpyDeviceToHost, stream_));
        TPA_CUDA(cudaEventRecord(ev1_, stream_));
        TPA_CUDA(cudaStreamSynchronize(stream_));
        TPA_CUDA(cudaGetLastError());
        int bodies = 0;
        bool more = false;
        for (int k = 0; k < K; ++k) {
            if (first && hs[k].skip) run[size_t(k)] = 0;
            if (!run[size_t(k)]) continue;
            bodies = std::max(bodies, hs[k].niter + ((hs[k].flags & 2) ? 1 : 0));
            stats[size_t(k)].restarts += 1;
            const double cur = hs[k].fin[1];
            if (cur <= guarded(k, cur) || !std::isfinite(cur) || hs[k].niter == 0 || hs[k].total >= max_cycles)
                run[size_t(k)] = 0;
            more = more || run[size_t(k)];
        }
        launches_ += bodies * body_launches_[precision];
        if (!more) break;
        TPA_CUDA(cudaMemcpyAsync(again_.p, run.data(), size_t(K) * sizeof(int), cudaMemcpyHostToDevice, stream_));
        plain(bk_restart, (K + 255) / 256, 256, 0, K, (const int*)again_.p, S, active_.p);
        ++launches_;
    }
    float ms = 0;
    cudaEventElapsedTime(&ms, ev0_, ev1_);
    for (int k = 0; k < K; ++k) {
        SolveStats& s = stats[size_t(k)];
        const double tv = total_volume(k), cur = hs[k].fin[1], tg = guarded(k, cur);
        auto l2 = [&](double sum) { return tv > 0 ? std::sqrt(sum / tv) : 0.0; };
        if (!hs[k].ok) {
            status[size_t(k)] = 1;
            messages[size_t(k)] = "Poisson right-hand side has nonzero volume mean";
        } else if (comp_vol_[size_t(k)] > 0) {
            s.removed_rhs_mean = hs[k].mb;
            s.removed_max_component_mean = std::fabs(hs[k].mb);
        }
        s.cycles = hs[k].total;
        s.converged = hs[k].ok && std::isfinite(cur) && std::isfinite(tg) && cur <= tg;
        s.initial_l2 = l2(hs[k].init[0]);
        s.initial_linf = hs[k].init[1];
        s.final_l2 = l2(hs[k].fin[0]);
        s.final_linf = cur;
        s.target_linf = tg;
        s.residual_scale = std::max(hs[k].init[1], kEps);
        s.ms_total = ms;
    }
    last_ms_ = ms;
}

double BatchSolver::total_volume(int k) const {
    return total_vol_.empty() ? 0.0 : total_vol_[size_t(k)];
}

template void BatchSolver::enqueue_vcycle<double>(const double*, int);
template void BatchSolver::enqueue_vcycle<float>(const double*, int);

}  // namespace tpa
