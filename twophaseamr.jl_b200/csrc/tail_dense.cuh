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
// MB at 2048, about the time of the multi-CTA launches a smaller tail would
// add) and, at any size that the set-up's shared memory holds, when the tail is
// the coarsest level alone, whose dense inverse has n^2 entries already.
#pragma once

#include "fused.cuh"

namespace tpa {

constexpr int kDenseTailCells = 2048;
constexpr int kDenseBuildThreads = 512;
constexpr int kDenseRows = 8;  // rows (warps) per CTA of the product

// Shared memory of the set-up for `C` unit vectors: right-hand side and iterate
// per level, two scratch vectors of the tail's first level.
inline size_t dense_build_smem(const std::vector<LevelView<double>>& v, int first, int C) {
    size_t cells = 2 * size_t(v[size_t(first)].n);
    for (size_t l = size_t(first); l < v.size(); ++l) cells += 2 * size_t(v[l].n);
    return cells * size_t(C) * sizeof(double);
}

// Columns C blockIdx.x .. of M (row-major, row stride ld): the tail's levels
// first..nl-1 applied to unit vectors held in shared memory, entry (i, c) of a
// vector at i C + c.  A thread takes a row for all C columns.  The phases and
// their arithmetic are those of tail_run.  remove_mean: the finest level's
// result without its volume mean (the whole hierarchy lies in the tail).
template <int C>
__global__ void __launch_bounds__(kDenseBuildThreads)
    k_dense_tail_build(const LevelView<double>* __restrict__ levels, int first, int nl, const double* __restrict__ G,
                       int gn, int remove_mean, double* __restrict__ M, int ld) {
    extern __shared__ double dense_sm[];
    __shared__ double mean[C];
    const int n0 = levels[first].n, col0 = blockIdx.x * C;
    const int tid = threadIdx.x, nt = blockDim.x;
    size_t cells = 0;
    for (int l = first; l < nl; ++l) cells += 2 * size_t(levels[l].n);
    double* u = dense_sm + cells * C;
    double* v = u + size_t(n0) * C;
    // mean[c] = scale * sum_i w_i a_ic (w null: 1)
    auto means = [&](const double* a, const double* w, int n, double scale) {
        for (int c = 0; c < C; ++c) {
            double s = 0;
            for (int i = tid; i < n; i += nt) s += w ? w[i] * a[i * C + c] : a[i * C + c];
            s = block_sum_all(s);
            if (tid == 0) mean[c] = s * scale;
        }
        __syncthreads();
    };
    auto rowdot = [&](const LevelView<double>& L, const double* a, int i, double (&acc)[C]) {
        for (int c = 0; c < C; ++c) acc[c] = 0;
        for (int k = L.rp[i]; k < L.rp[i + 1]; ++k) {
            const double av = L.val[k];
            const double* aj = a + size_t(L.ci[k]) * C;
            for (int c = 0; c < C; ++c) acc[c] += av * aj[c];
        }
    };
    double* bp = dense_sm;
    for (int e = tid; e < n0 * C; e += nt) bp[e] = (e / C == col0 + e % C) ? 1.0 : 0.0;
    __syncthreads();
    for (int l = first;; ++l) {
        const LevelView<double> L = with_weights(levels[l]);
        double* x = bp + size_t(L.n) * C;
        if (L.singular) {
            means(bp, nullptr, L.n, L.cvol_inv);
            for (int e = tid; e < L.n * C; e += nt) bp[e] -= L.vol[e / C] * mean[e % C];
            __syncthreads();
        }
        double acc[C];
        if (l == nl - 1) {
            const int lane = tid & 31;
            for (int i = tid >> 5; i < gn; i += nt >> 5) {
                for (int c = 0; c < C; ++c) acc[c] = 0;
                for (int k = lane; k < gn; k += 32) {
                    const double g = G[size_t(i) * gn + k];
                    for (int c = 0; c < C; ++c) acc[c] += g * bp[k * C + c];
                }
                for (int c = 0; c < C; ++c) {
                    for (int o = 16; o; o >>= 1) acc[c] += __shfl_down_sync(0xffffffffu, acc[c], o);
                    if (!lane) x[i * C + c] = acc[c];
                }
            }
            __syncthreads();
            break;
        }
        for (int e = tid; e < L.n * C; e += nt) u[e] = L.w * L.dinv[e / C] * bp[e];
        __syncthreads();
        for (int i = tid; i < L.n; i += nt) {
            rowdot(L, u, i, acc);
            for (int c = 0; c < C; ++c) x[i * C + c] = u[i * C + c] + L.w * L.dinv[i] * (bp[i * C + c] - acc[c]);
        }
        __syncthreads();
        for (int i = tid; i < L.n; i += nt) {
            rowdot(L, x, i, acc);
            for (int c = 0; c < C; ++c) {
                const double r = bp[i * C + c] - acc[c];
                v[i * C + c] = r;
                u[i * C + c] = L.tinv[i] * r;
            }
        }
        __syncthreads();
        double* bc = x + size_t(L.n) * C;  // the next level's right-hand side
        for (int J = tid; J < L.nc; J += nt) {
            double sum[C];
            for (int c = 0; c < C; ++c) sum[c] = 0;
            for (int k = L.cptr[J]; k < L.cptr[J + 1]; ++k) {
                const int i = L.child[k];
                rowdot(L, u, i, acc);
                for (int c = 0; c < C; ++c) sum[c] += v[i * C + c] - L.tw * acc[c];
            }
            for (int c = 0; c < C; ++c) bc[J * C + c] = sum[c];
        }
        __syncthreads();
        bp = bc;
    }
    for (int l = nl - 2; l >= first; --l) {
        const LevelView<double> L = with_weights(levels[l]);
        const double* xc = bp + size_t(levels[l + 1].n) * C;
        bp -= 2 * size_t(L.n) * C;
        double* x = bp + size_t(L.n) * C;
        double acc[C];
        for (int e = tid; e < L.n * C; e += nt) u[e] = xc[L.owner[e / C] * C + e % C];
        __syncthreads();
        for (int i = tid; i < L.n; i += nt) {
            rowdot(L, u, i, acc);
            for (int c = 0; c < C; ++c) x[i * C + c] += u[i * C + c] - L.tw * L.tinv[i] * acc[c];
        }
        __syncthreads();
        for (int sweep = 0; sweep < 2; ++sweep) {
            const double* in = sweep ? v : x;
            double* out = sweep ? x : v;
            for (int i = tid; i < L.n; i += nt) {
                rowdot(L, in, i, acc);
                for (int c = 0; c < C; ++c)
                    out[i * C + c] = in[i * C + c] + L.w * L.dinv[i] * (bp[i * C + c] - acc[c]);
            }
            __syncthreads();
        }
    }
    double* x = bp + size_t(n0) * C;
    if (remove_mean) {
        means(x, levels[first].vol, n0, levels[first].cvol_inv);
        for (int e = tid; e < n0 * C; e += nt) x[e] -= mean[e % C];
        __syncthreads();
    }
    for (int e = tid; e < n0 * C; e += nt)
        if (col0 + e % C < n0) M[size_t(e / C) * ld + col0 + e % C] = x[e];
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
