// The coarse tail as one dense product.
//
// Everything below the multi-CTA levels -- the tail's sweeps, transfers,
// right-hand-side projections and the dense coarse solve -- is one linear map
// x = M b from the tail's right-hand side to its correction (the cycle of
// src/solvers/multigrid/cycles.jl:46-77 of ronaldremmerswaal/TwoPhaseAMR.jl is
// linear: damped Jacobi from zero, fixed transfers, a fixed coarse inverse).
// `k_dense_tail_build` forms M once per hierarchy and refresh, by running the
// tail on the unit vectors in FP64; a V-cycle then applies it in one launch
// over the whole chip (`k_tail_dense`).
//
// Why: walking the tail's phases in one CTA is a chain of dependent global
// loads and CTA barriers, about 20 us for levels of 1024 and 256 cells, 30 us
// for three levels and 37 us for 2048 + 512 cells, with 147 SMs idle.  The
// product reads 8 n^2 bytes (8.4 MB at n = 1024, held in L2), one row per warp,
// and its loads of M do not depend on the kernels before it, so they are issued
// before the programmatic-launch wait.  Measured per solve, start against here:
// 32^2 box 534 -> 365 us, periodic 128^2 913 -> 724, 1024 x 512 (2048-cell tail)
// 1581 -> 1321, droplet of 110k cells 1955 -> 1707 us.
//
// The map is used for tails of at most kDenseTailCells cells (n^2 doubles: 32
// MB at 2048) and, at any size, when the tail is the coarsest level alone, whose
// dense inverse has n^2 entries already: at most 8191 cells (hierarchy.cpp), where
// the map takes another 537 MB and one unit vector 131 KB of shared memory.
// At 2048 + 512 cells against a tail of 512 below two launches of the 2048-cell
// level: solves of 64 x 32 to 1024 x 512 periodic cells 0-8 % slower mixed (325
// and 300 us at 128 x 64), 0-8 % FP64, and 256 x 128 walled cells on tiles 473 and
// 459 us; a refresh that forms the map 776 and 549 us.  The walked tail of that
// size takes 37 us a V-cycle in place of 9.
#pragma once

#include "fused.cuh"

namespace tpa {

constexpr int kDenseTailCells = 2048;
constexpr int kDenseBuildThreads = 512;
constexpr int kDenseRows = 8;  // rows (warps) per CTA of the product

// Shared memory of the set-up for `C` unit vectors: a right-hand side and an
// iterate per level, the first level's right-hand side (known in closed form)
// giving its place to a scratch vector.
inline size_t dense_build_smem(const std::vector<LevelView<double>>& v, int first, int C) {
    size_t cells = 0;
    for (size_t l = size_t(first); l < v.size(); ++l) cells += 2 * size_t(v[l].n);
    return cells * size_t(C) * sizeof(double);
}

// Columns C blockIdx.x .. of M (row-major, row stride ld): the tail's levels
// first..nl-1 applied to unit vectors held in shared memory, one behind the
// other.  A thread takes rows tid + q kDenseBuildThreads, q < ROWS,
// for all C columns.  The phases and their arithmetic are those of tail_run.
// remove_mean: the finest level's result without its volume mean (the whole
// hierarchy lies in the tail).
//
// Bound by the latency of a phase's loads, nine phases a level.  So a level's
// operator rows are loaded once for its downward and once for its upward phases
// (kHeld entries, a lattice row's, in registers), which leaves the phases with
// shared memory alone; a row's restriction is formed by the row's own thread;
// and C is as large as lets all columns run at once (128 CTAs of 8 columns at
// 1024 cells).  The columns lie one behind the other: side by side, a warp's
// loads fall on a quarter of the banks.  At 1024 + 256 cells 134 us with four
// columns a CTA and every phase's operator read from L2, 61 us so.
template <int C, int ROWS>
__global__ void __launch_bounds__(kDenseBuildThreads, 1)
    k_dense_tail_build(const LevelView<double>* __restrict__ levels, int first, int nl, const double* __restrict__ G,
                       int gn, int remove_mean, double* __restrict__ M, int ld) {
    constexpr int NT = kDenseBuildThreads, kHeld = 5, kG = 4;
    extern __shared__ __align__(16) double dense_sm[];
    __shared__ double mean[C];
    const int n0 = levels[first].n, col0 = blockIdx.x * C;
    const int tid = threadIdx.x;
    double* const u = dense_sm;  // scratch; the right-hand side when the first level is the last
    // mean[c] = scale * sum_i w_i a_ic (w null: 1)
    auto means = [&](const double* a, const double* w, int n, double scale) {
        for (int c = 0; c < C; ++c) {
            double s = 0;
            for (int i = tid; i < n; i += NT) s += w ? w[i] * a[c * n + i] : a[c * n + i];
            s = block_sum_all(s);
            if (tid == 0) mean[c] = s * scale;
        }
        __syncthreads();
    };
    // row i of a level's vectors (n rows)
    struct Cols {
        double v[C];
    };
    auto get = [](const double* a, int i, int n) {
        Cols o;
#pragma unroll
        for (int c = 0; c < C; ++c) o.v[c] = a[c * n + i];
        return o;
    };
    auto put = [](double* a, int i, int n, const Cols& o) {
#pragma unroll
        for (int c = 0; c < C; ++c) a[c * n + i] = o.v[c];
    };
    auto project = [&](const LevelView<double>& L, double* b) {
        for (int i = tid; i < L.n; i += NT)
            for (int c = 0; c < C; ++c) b[c * L.n + i] -= L.vol[i] * mean[c];
        __syncthreads();
    };
    // this thread's rows of a level
    double held[ROWS][kHeld];
    unsigned col[ROWS][(kHeld + 1) / 2];  // two columns a word
    int width[ROWS];
    auto load_rows = [&](const LevelView<double>& L) {
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
            const int i = tid + q * NT;
            width[q] = 0;
            if (i >= L.n) continue;
            const int k0 = L.rp[i];
            width[q] = L.rp[i + 1] - k0;
#pragma unroll
            for (int k = 0; k < kHeld; ++k) held[q][k] = k < width[q] ? L.val[k0 + k] : 0.0;
#pragma unroll
            for (int k = 0; k < kHeld; k += 2) {
                const unsigned a = k < width[q] ? unsigned(L.ci[k0 + k]) : 0u;
                const unsigned b = k + 1 < kHeld && k + 1 < width[q] ? unsigned(L.ci[k0 + k + 1]) : 0u;
                col[q][k / 2] = a | b << 16;
            }
        }
    };
    auto rowdot = [&](const LevelView<double>& L, const double* a, int q) {
        Cols acc;
#pragma unroll
        for (int c = 0; c < C; ++c) acc.v[c] = 0;
#pragma unroll
        for (int k = 0; k < kHeld; ++k)
            if (k < width[q]) {
                const unsigned j = k % 2 ? col[q][k / 2] >> 16 : col[q][k / 2] & 0xffffu;
                const Cols t = get(a, int(j), L.n);
#pragma unroll
                for (int c = 0; c < C; ++c) acc.v[c] += held[q][k] * t.v[c];
            }
        if (width[q] > kHeld) {
            const int k0 = L.rp[tid + q * NT];
            for (int k = kHeld; k < width[q]; ++k) {
                const double w = L.val[k0 + k];
                const Cols t = get(a, L.ci[k0 + k], L.n);
#pragma unroll
                for (int c = 0; c < C; ++c) acc.v[c] += w * t.v[c];
            }
        }
        return acc;
    };
    // right-hand side row i of the first level: the unit vectors, projected (the
    // columns past n0 are not stored)
    const double mean0 = levels[first].cvol_inv;
    auto rhs0 = [&](const LevelView<double>& L, int i) {
        Cols o;
        const double vol = L.singular ? L.vol[i] : 0.0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            o.v[c] = i == col0 + c ? 1.0 : 0.0;
            if (L.singular) o.v[c] -= vol * mean0;
        }
        return o;
    };
    double* bp = u;                      // level's right-hand side; the first level's lies nowhere
    double* x = u + size_t(n0) * C;
    for (int l = first;; ++l) {
        const LevelView<double> L = with_weights(levels[l]);
        if (l == nl - 1) {
            if (l == first) {
                for (int i = tid; i < n0; i += NT) put(bp, i, n0, rhs0(L, i));
                __syncthreads();
            } else if (L.singular) {
                means(bp, nullptr, L.n, L.cvol_inv);
                project(L, bp);
            }
            // kG rows of the inverse at once, so that a value of bp is read once for them
            const int lane = tid & 31;
            for (int i = kG * (tid >> 5); i < gn; i += kG * (NT >> 5)) {
                Cols acc[kG];
#pragma unroll
                for (int k = 0; k < kG; ++k)
#pragma unroll
                    for (int c = 0; c < C; ++c) acc[k].v[c] = 0;
#pragma unroll 2
                for (int j = lane; j < gn; j += 32) {
                    double g[kG];
#pragma unroll
                    for (int k = 0; k < kG; ++k) g[k] = G[size_t(min(i + k, gn - 1)) * gn + j];
                    const Cols t = get(bp, j, gn);
#pragma unroll
                    for (int k = 0; k < kG; ++k)
#pragma unroll
                        for (int c = 0; c < C; ++c) acc[k].v[c] += g[k] * t.v[c];
                }
#pragma unroll
                for (int k = 0; k < kG; ++k) {
#pragma unroll
                    for (int c = 0; c < C; ++c)
                        for (int o = 16; o; o >>= 1) acc[k].v[c] += __shfl_down_sync(0xffffffffu, acc[k].v[c], o);
                    if (!lane && i + k < gn) put(x, i + k, gn, acc[k]);
                }
            }
            __syncthreads();
            break;
        }
        load_rows(L);
        if (l > first && L.singular) {
            means(bp, nullptr, L.n, L.cvol_inv);
            project(L, bp);
        }
        auto rhs = [&](int i) { return l == first ? rhs0(L, i) : get(bp, i, L.n); };
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
            const int i = tid + q * NT;
            if (i >= L.n) continue;
            Cols t = rhs(i);
            const double d = L.w * L.dinv[i];
#pragma unroll
            for (int c = 0; c < C; ++c) t.v[c] = d * t.v[c];
            put(u, i, L.n, t);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
            const int i = tid + q * NT;
            if (i >= L.n) continue;
            const Cols acc = rowdot(L, u, q), b = rhs(i);
            Cols t = get(u, i, L.n);
            const double d = L.w * L.dinv[i];
#pragma unroll
            for (int c = 0; c < C; ++c) t.v[c] += d * (b.v[c] - acc.v[c]);
            put(x, i, L.n, t);
        }
        __syncthreads();
        Cols r[ROWS];
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
            const int i = tid + q * NT;
            if (i >= L.n) continue;
            const Cols acc = rowdot(L, x, q);
            r[q] = rhs(i);
            Cols t;
            const double d = L.tinv[i];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                r[q].v[c] -= acc.v[c];
                t.v[c] = d * r[q].v[c];
            }
            put(u, i, L.n, t);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
            if (tid + q * NT >= L.n) continue;
            const Cols acc = rowdot(L, u, q);
#pragma unroll
            for (int c = 0; c < C; ++c) r[q].v[c] -= L.tw * acc.v[c];
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < ROWS; ++q)
            if (tid + q * NT < L.n) put(u, tid + q * NT, L.n, r[q]);
        __syncthreads();
        double* bc = x + size_t(L.n) * C;  // the next level's right-hand side
        for (int J = tid; J < L.nc; J += NT) {
            Cols sum;
#pragma unroll
            for (int c = 0; c < C; ++c) sum.v[c] = 0;
            for (int k = L.cptr[J]; k < L.cptr[J + 1]; ++k) {
                const Cols t = get(u, L.child[k], L.n);
#pragma unroll
                for (int c = 0; c < C; ++c) sum.v[c] += t.v[c];
            }
            put(bc, J, L.nc, sum);
        }
        __syncthreads();
        bp = bc;
        x = bc + size_t(L.nc) * C;
    }
    for (int l = nl - 2; l >= first; --l) {
        const LevelView<double> L = with_weights(levels[l]);
        load_rows(L);
        const double* xc = x;
        x = bp - size_t(L.n) * C;
        bp = l == first ? u : x - size_t(L.n) * C;
        auto rhs = [&](int i) { return l == first ? rhs0(L, i) : get(bp, i, L.n); };
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
            const int i = tid + q * NT;
            if (i < L.n) put(u, i, L.n, get(xc, L.owner[i], levels[l + 1].n));
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
            const int i = tid + q * NT;
            if (i >= L.n) continue;
            const Cols acc = rowdot(L, u, q), t = get(u, i, L.n);
            Cols o = get(x, i, L.n);
            const double d = L.tw * L.tinv[i];
#pragma unroll
            for (int c = 0; c < C; ++c) o.v[c] += t.v[c] - d * acc.v[c];
            put(x, i, L.n, o);
        }
        __syncthreads();
        for (int sweep = 0; sweep < 2; ++sweep) {
            const double* in = sweep ? u : x;
            double* out = sweep ? x : u;
#pragma unroll
            for (int q = 0; q < ROWS; ++q) {
                const int i = tid + q * NT;
                if (i >= L.n) continue;
                const Cols acc = rowdot(L, in, q), b = rhs(i);
                Cols o = get(in, i, L.n);
                const double d = L.w * L.dinv[i];
#pragma unroll
                for (int c = 0; c < C; ++c) o.v[c] += d * (b.v[c] - acc.v[c]);
                put(out, i, L.n, o);
            }
            __syncthreads();
        }
    }
    if (remove_mean) {
        means(x, levels[first].vol, n0, levels[first].cvol_inv);
        for (int i = tid; i < n0; i += NT)
            for (int c = 0; c < C; ++c) x[c * n0 + i] -= mean[c];
        __syncthreads();
    }
    for (int e = tid; e < n0 * C; e += NT)
        if (col0 + e % C < n0) M[size_t(e / C) * ld + col0 + e % C] = x[(e % C) * n0 + e / C];
}

// x = M b: a warp per row, the row's first 1024 entries in flight before the
// wait (M is written by set-up only, and the host waits for it before any
// V-cycle is launched), b staged in shared memory once per CTA.  mean_out (may
// be null): the whole hierarchy is the tail and M removes the mean itself; the
// CG's epilogue then takes r'x.
// Bound by the latency of one launch, the load of b and the warp sum.
template <typename T, typename TB, typename Epi>
__global__ void __launch_bounds__(32 * kDenseRows)
    k_tail_dense(int n, int ld, const double* __restrict__ M, const TB* b, T* x, double* mean_out,
                 unsigned* counter, Epi epi) {
    pdl_launch();
    constexpr int kChunk = 2048;
    __shared__ __align__(16) double sb[kChunk];
    const int lane = threadIdx.x & 31, row = blockIdx.x * kDenseRows + (threadIdx.x >> 5);
    const double* m = M + size_t(row < n ? row : 0) * ld;
    double2 t[16];
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int k = k0 + 64 * q + 2 * lane;
            t[q] = k < n ? ld_static(reinterpret_cast<const double2*>(m + k)) : make_double2(0.0, 0.0);
        }
    };
    load(0);
    pdl_wait();
    double acc[4] = {0, 0, 0, 0};
    for (int k0 = 0; k0 < n; k0 += 1024) {
        if (k0 % kChunk == 0) {
            if (k0) __syncthreads();
            const int count = min(kChunk, (n - k0 + 1) & ~1);
            for (int i = threadIdx.x; i < count; i += blockDim.x) sb[i] = k0 + i < n ? double(b[k0 + i]) : 0.0;
            __syncthreads();
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int k = k0 + 64 * q + 2 * lane;
            if (k < n) {
                const double2 bb = *reinterpret_cast<const double2*>(sb + k % kChunk);
                acc[(2 * q) & 3] += t[q].x * bb.x;
                acc[(2 * q + 1) & 3] += t[q].y * bb.y;
            }
        }
        if (k0 + 1024 < n) load(k0 + 1024);
    }
    double s = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (!lane && row < n) x[row] = T(s);
    if (mean_out && blockIdx.x == 0 && threadIdx.x == 0) *mean_out = 0.0;
    if constexpr (Epi::kRz) {
        const double rx = !lane && row < n ? double(epi.r[row]) * double(T(s)) : 0.0;
        fold_sum(rx, epi.partial, counter, [&](double t) { epi(0.0, t); });
    }
}

}  // namespace tpa
