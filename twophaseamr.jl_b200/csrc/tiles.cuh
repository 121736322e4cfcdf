// Fused per-level V-cycle kernels on haloed block tiles (tiles.hpp).
//
// A level of the default cycle (damped Jacobi, two pre- and two post-sweeps,
// src/solvers/multigrid/cycles.jl:8-77 of ronaldremmerswaal/TwoPhaseAMR.jl)
// costs six dependent launches on the unfused path (k_pre2, k_residual,
// k_restrict, k_prolong, k_post1, k_post2).  Here one CTA owns one block and
// recomputes the values its block needs from a halo of three rings, so a
// level costs two launches:
//   k_tile_down  rings <= 3: x1 = w D^-1 bp (the first sweep from zero);
//                rings <= 2: x2 = x1 + w D^-1 (bp - A x1);
//                rings <= 1: r = bp - A x2, s = Dt^-1 r;
//                the block:  b_c = P_tent'(r - wt A s) for its coarse cells,
//                            x2 and bp stored (x2 into L.y)
//   k_tile_up    rings <= 3: e = x_c(owner);
//                rings <= 2: x = x2 + e - wt Dt^-1 A e;
//                rings <= 1: x' = x + w D^-1 (bp - A x);
//                the block:  x'' = x' + w D^-1 (bp - A x') into L.x, the
//                            finest level's mean (and epilogue)
// Every row is summed in CSR order with the arithmetic of the unfused kernels
// (pre2_cell, residual_cell, restrict_quad, prolong_cell, sweep_cell), so the
// two paths give the same V-cycle up to rounding.
//
// A thread owns one row of the tile (two on tiles of more than 1024 rows): it
// holds the row's entries, right-hand side, diagonals and iterate in registers
// through all phases, and only the vector that a phase reads at other rows
// goes through shared memory.  A row's products load independent shared-memory
// words, where walking a staged CSR row was a chain of dependent loads; per
// tile of a 16 x 16 block this is about 2.4 k warp instructions in place of 14 k.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "fused.cuh"
#include "stencil.cuh"
#include "tiles.hpp"

namespace tpa {

constexpr int kTileThreads = 256;  // stencil tiles
constexpr int kTileMaxCells = 1536;  // cells of a CSR tile (rings <= 3) at most

// One level's tiles in precision T (device pointers).
template <typename T>
struct TileView {
    const TileInfo* info;
    const int* cell;
    const int* own;     // parallel to cell: tentative owner on the coarse level
    const int2* slice;  // {first entry, width}
    const T* val;       // the level's operator values in entry order (0: padding)
    const short* col;
    const int* co;
    const short4* ch;   // per coarse cell: local indices of its children (-1: none)
};

// threads of a tile: one per `rows` rows and per rows + 1 cells
inline int tile_threads(int n3max, int n2max, int rows) {
    const int by_rows = (n2max + rows - 1) / rows, by_cells = (n3max + rows) / (rows + 1);
    return ((by_rows > by_cells ? by_rows : by_cells) + 31) & ~31;
}

// Kernel forms of a level's CSR tiles by the threads a tile takes (a thread per
// row, rounded to warps): launch bounds that leave FP64 rows their registers on
// 8 x 8 and 16 x 16 blocks, and two rows per thread beyond 1024.
template <typename F>
void with_tile_threads(int threads, int rows, F f) {
    if (rows == 2) f(std::integral_constant<int, 1024>(), std::integral_constant<int, 2>());
    else if (threads <= 256) f(std::integral_constant<int, 256>(), std::integral_constant<int, 1>());
    else if (threads <= 640) f(std::integral_constant<int, 640>(), std::integral_constant<int, 1>());
    else f(std::integral_constant<int, 1024>(), std::integral_constant<int, 1>());
}

// The three vectors that rows read from one another, at offsets known to the
// compiler: cells (rings <= 3), then two of the rows.
template <typename T, int NT, int ROWS>
struct TileShared {
    static constexpr int kCells = (ROWS + 1) * NT < kTileMaxCells ? (ROWS + 1) * NT : kTileMaxCells;
    static constexpr int kRows = ROWS * NT < kTileMaxCells ? ROWS * NT : kTileMaxCells;
    T a[kCells], b[kRows], c[kRows];
};

__device__ __forceinline__ TileInfo tile_info(const TileInfo* p) {
    const int4* q = reinterpret_cast<const int4*>(p);
    const int4 a = ld_static(q), b = ld_static(q + 1);
    return TileInfo{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}

// a row's entries in registers (w: its slice's width, the same over the warp)
template <typename T>
struct TileRow {
    T v[kTileMaxRow];
    int c[kTileMaxRow];
    int w;
    __device__ __forceinline__ void load(const TileView<T>& V, int first, int k, int n2) {
        w = 0;
        if (k - (k & 31) >= n2) return;  // a slice beyond the tile's rows (whole warps)
        const int2 s = ld_static(V.slice + first + (k >> 5));
        w = s.y;
        const T* val = V.val + s.x + (k & 31);
        const short* col = V.col + s.x + (k & 31);
#pragma unroll
        for (int u = 0; u < kTileMaxRow; ++u) {
            if (u < w) {
                v[u] = ld_static(val + 32 * u);
                c[u] = ld_static(col + 32 * u);
            }
        }
    }
    __device__ __forceinline__ T dot(const T* x) const {
        T acc = T(0);
#pragma unroll
        for (int u = 0; u < kTileMaxRow; ++u)
            if (u < w) acc += v[u] * x[c[u]];
        return acc;
    }
};

// Right-hand side of a level of one solve: the level's own or, on the finest
// level, the caller's residual (FP64 or FP32), projected by the level's sum.
template <typename TB>
struct TileRhs {
    const TB* b;
    const double* sum;  // null: not projected
    template <typename T>
    __device__ __forceinline__ bool projects(const LevelView<T>& L) const {
        return L.singular && sum;
    }
    template <typename T>
    __device__ __forceinline__ bool start(const LevelView<T>& L, double& mean) const {
        mean = projects(L) ? *sum * L.cvol_inv : 0.0;
        return true;
    }
    __device__ __forceinline__ TB load(int g) const { return b[g]; }
};

// The down half on tile blockIdx.x: src gives the right-hand side; bc receives
// the coarse one; bp_out (null: not written, the cycle reads b itself) the
// projected right-hand side for the up half; the pre-smoothed iterate goes to
// L.y.  ROWS rows and ROWS + 1 cells per thread.
template <typename T, int NT, int ROWS, typename Src>
__device__ __forceinline__ void tile_down(const LevelView<T>& L, const TileView<T>& V, const Src& src,
                                          T* bc, T* bp_out) {
    __shared__ TileShared<T, NT, ROWS> sm;
    T *xa = sm.a, *xb = sm.b, *ss = sm.c;
    constexpr int CU = ROWS + 1;
    const TileInfo I = tile_info(V.info + blockIdx.x);
    const int nt = blockDim.x;
    int g[CU];
#pragma unroll
    for (int u = 0; u < CU; ++u) {
        const int k = threadIdx.x + u * nt;
        g[u] = k < I.n3 ? ld_static(V.cell + I.cell + k) : -1;
    }
    TileRow<T> row[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) row[q].load(V, I.slice, threadIdx.x + q * nt, I.n2);
    const bool project = src.projects(L);
    T vv[CU], dd[CU], tt[ROWS];
#pragma unroll
    for (int u = 0; u < CU; ++u) {
        vv[u] = dd[u] = T(0);
        if (g[u] >= 0) {
            if (project) vv[u] = ld_static(L.vol + g[u]);
            dd[u] = ld_static(L.dinv + g[u]);
        }
    }
#pragma unroll
    for (int q = 0; q < ROWS; ++q) tt[q] = int(threadIdx.x) + q * nt < I.n1 ? ld_static(L.tinv + g[q]) : T(0);
    short4 ch0 = make_short4(-1, -1, -1, -1);
    int co0 = 0;
    if (int(threadIdx.x) < I.nco) {
        ch0 = ld_static(V.ch + I.co + threadIdx.x);
        co0 = ld_static(V.co + I.co + threadIdx.x);
    }
    pdl_wait();
    double mean;
    if (!src.start(L, mean)) return;  // the same over the tile
    T bp[CU];
#pragma unroll
    for (int u = 0; u < CU; ++u)
        if (g[u] >= 0) {
            double v = double(src.load(g[u]));
            if (project) v -= double(vv[u]) * mean;  // as proj_b
            bp[u] = T(v);
        }
    T xr[ROWS], rr[ROWS];
#pragma unroll
    for (int u = 0; u < CU; ++u)
        if (g[u] >= 0) {
            const T x1 = L.w * dd[u] * bp[u];
            xa[threadIdx.x + u * nt] = x1;
            if (u < ROWS) xr[u] = x1;
        }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int k = threadIdx.x + q * nt;
        if (k < I.n2) {
            xr[q] = xr[q] + L.w * dd[q] * (bp[q] - row[q].dot(xa));
            xb[k] = xr[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int k = threadIdx.x + q * nt;
        if (k < I.n1) {
            rr[q] = bp[q] - row[q].dot(xb);
            ss[k] = tt[q] * rr[q];
        }
        if (k < I.n0) {
            L.y[g[q]] = xr[q];  // the pre-smoothed iterate, read by the up half
            if (bp_out) bp_out[g[q]] = bp[q];
        }
    }
    __syncthreads();
    T* t = xa;  // r - wt A s on the block
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int k = threadIdx.x + q * nt;
        if (k < I.n0) t[k] = rr[q] - L.tw * row[q].dot(ss);
    }
    __syncthreads();
    // a coarse cell per thread, its children in the fixed order (c0 + c1) + (c2 + c3)
    for (int J = threadIdx.x; J < I.nco; J += nt) {
        const short4 c = J == int(threadIdx.x) ? ch0 : V.ch[I.co + J];
        const T c0 = c.x >= 0 ? t[c.x] : T(0), c1 = c.y >= 0 ? t[c.y] : T(0);
        const T c2 = c.z >= 0 ? t[c.z] : T(0), c3 = c.w >= 0 ? t[c.w] : T(0);
        bc[J == int(threadIdx.x) ? co0 : V.co[I.co + J]] = (c0 + c1) + (c2 + c3);
    }
}

// The up half: xc the coarse level's correction, bp_in the projected right-hand
// side; out(g, x) takes the result of cell g and its value from `pre(g)`, which
// is called before the wait (static data) and `late(g)` after it.
template <typename T, int NT, int ROWS, typename Out>
__device__ __forceinline__ void tile_up(const LevelView<T>& L, const TileView<T>& V, const T* xc, const T* bp_in,
                                        Out& out) {
    __shared__ TileShared<T, NT, ROWS> sm;
    T *e = sm.a, *xp = sm.b, *xq = sm.c;
    constexpr int CU = ROWS + 1;
    const TileInfo I = tile_info(V.info + blockIdx.x);
    const int nt = blockDim.x;
    int g[CU], o[CU];
#pragma unroll
    for (int u = 0; u < CU; ++u) {
        const int k = threadIdx.x + u * nt;
        g[u] = k < I.n3 ? ld_static(V.cell + I.cell + k) : -1;
        o[u] = k < I.n3 ? ld_static(V.own + I.cell + k) : -1;
    }
    TileRow<T> row[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) row[q].load(V, I.slice, threadIdx.x + q * nt, I.n2);
    T dd[ROWS], tt[ROWS], x[ROWS], bb[ROWS], er[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int k = threadIdx.x + q * nt;
        if (k < I.n2) {
            dd[q] = ld_static(L.dinv + g[q]);
            tt[q] = ld_static(L.tinv + g[q]);
        }
        out.before(q, g[q], k < I.n0);
    }
    pdl_wait();
    if (!out.start()) return;  // the same over the tile
#pragma unroll
    for (int u = 0; u < CU; ++u) {
        const int k = threadIdx.x + u * nt;
        if (g[u] >= 0) {
            const T ev = xc[o[u]];
            e[k] = ev;
            if (u < ROWS) er[u] = ev;
        }
    }
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int k = threadIdx.x + q * nt;
        if (k < I.n2) x[q] = L.y[g[q]];
        if (k < I.n1) bb[q] = bp_in[g[q]];
        out.after(q, g[q], k < I.n0);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int k = threadIdx.x + q * nt;
        if (k < I.n2) {
            x[q] += er[q] - L.tw * tt[q] * row[q].dot(e);
            xp[k] = x[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int k = threadIdx.x + q * nt;
        if (k < I.n1) {
            x[q] = x[q] + L.w * dd[q] * (bb[q] - row[q].dot(xp));
            xq[k] = x[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
        const int k = threadIdx.x + q * nt;
        if (k < I.n0) {
            const T v = x[q] + L.w * dd[q] * (bb[q] - row[q].dot(xq));
            L.x[g[q]] = v;
            out.take(q, double(v));
        }
    }
}

template <typename T, typename TB, int NT, int ROWS>
__global__ void __launch_bounds__(NT, 1)
    k_tile_down(LevelView<T> L, TileView<T> V, TileRhs<TB> src, T* bc, T* bp_out) {
    pdl_launch();
    tile_down<T, NT, ROWS>(with_weights(L), V, src, bc, bp_out);
}

// What the up half of one solve's level does with its result: the sums of the
// finest level's mean (mean_out not null) and of the epilogue's r'x.
template <typename T, typename Epi, int ROWS>
struct TileMean {
    const T* vol;
    bool on;
    const Epi& epi;
    T vv[ROWS];
    double rv[ROWS];
    double v = 0, w = 0;
    __device__ __forceinline__ void before(int q, int g, bool own) {
        if (on && own) vv[q] = ld_static(vol + g);
    }
    __device__ __forceinline__ bool start() const { return true; }
    __device__ __forceinline__ void after(int q, int g, bool own) {
        if constexpr (Epi::kRz)
            if (on && own) rv[q] = double(epi.r[g]);
    }
    __device__ __forceinline__ void take(int q, double x) {
        if (!on) return;
        v += double(vv[q]) * x;
        if constexpr (Epi::kRz) w += rv[q] * x;
    }
};

// xc: the coarse level's correction; bp_in: the projected right-hand side (the
// level's own below the finest); mean_out (may be null): the volume mean of the
// result, folded by the last CTA, which then runs `epi`.
template <typename T, typename Epi, int NT, int ROWS>
__global__ void __launch_bounds__(NT, 1)
    k_tile_up(LevelView<T> L, TileView<T> V, const T* xc, const T* bp_in, double* partial, unsigned* counter,
              double* mean_out, Epi epi) {
    pdl_launch();
    TileMean<T, Epi, ROWS> out{L.vol, mean_out != nullptr, epi};
    tile_up<T, NT, ROWS>(with_weights(L), V, xc, bp_in, out);
    if (mean_out) fold_mean(out.v, out.w, partial, counter, mean_out, L.cvol_inv, epi);
}

// tile copies of a level's CSR values: out[k] = val[pos[k]] (0 for padding)
template <typename T>
__global__ void k_tile_gather(int m, const int* __restrict__ pos, const T* __restrict__ val, T* __restrict__ out) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x)
        out[k] = pos[k] >= 0 ? val[pos[k]] : T(0);
}

// ---------------------------------------------------------------------------------
// The same two launches per level on constant-coefficient 16x16 levels (the
// levels of the vectorized kernels, stencil4.cuh: every block and its
// neighbours the same size, every coupling c0): the tile is the block plus a
// three-cell frame, a 22 x 22 square taken from the block and its eight
// neighbours (W, E, S, N from the neighbour table, the corners through them;
// cells of missing blocks -- walls -- do not exist), with no index lists.
// Each phase works on a square one cell smaller than the last.  The row
// arithmetic is that of the vectorized kernels (q_apply: the existing
// neighbours summed west, east, south, north).

namespace vt {
constexpr int R = 22;  // region side: 16 + 2 * 3
__device__ __forceinline__ int at(int i, int j) { return (j + 3) * R + (i + 3); }
}  // namespace vt

// the nine blocks around block b (index (by + 1) * 3 + (bx + 1), -1: none)
template <typename T>
__device__ __forceinline__ void vt_blocks(const SView<T>& L, int b, int* nb9) {
    if (threadIdx.x == 0) {
        const int4 c = ld_static(reinterpret_cast<const int4*>(L.nbr + 4 * b));
        const int4 none = make_int4(-1, -1, -1, -1);
        const int4 w = c.x >= 0 ? ld_static(reinterpret_cast<const int4*>(L.nbr + 4 * c.x)) : none;
        const int4 e = c.y >= 0 ? ld_static(reinterpret_cast<const int4*>(L.nbr + 4 * c.y)) : none;
        const int4 s = c.z >= 0 ? ld_static(reinterpret_cast<const int4*>(L.nbr + 4 * c.z)) : none;
        const int4 n = c.w >= 0 ? ld_static(reinterpret_cast<const int4*>(L.nbr + 4 * c.w)) : none;
        nb9[0] = c.x >= 0 ? w.z : s.x;  // south-west
        nb9[1] = c.z;
        nb9[2] = c.y >= 0 ? e.z : s.y;  // south-east
        nb9[3] = c.x;
        nb9[4] = b;
        nb9[5] = c.y;
        nb9[6] = c.x >= 0 ? w.w : n.x;  // north-west
        nb9[7] = c.w;
        nb9[8] = c.y >= 0 ? e.w : n.y;  // north-east
    }
}

// global cell of region cell (i, j), i, j in [-3, 18], or -1 when it does not exist
__device__ __forceinline__ int vt_cell(const int* nb9, int i, int j) {
    const int bx = i < 0 ? -1 : (i > 15 ? 1 : 0), by = j < 0 ? -1 : (j > 15 ? 1 : 0);
    const int B = nb9[(by + 1) * 3 + bx + 1];
    if (B < 0) return -1;
    return B * 256 + (j - 16 * by) * 16 + (i - 16 * bx);
}

// c0 (count * v - sum of the existing neighbours), neighbours in the order of q_apply
template <typename T>
__device__ __forceinline__ T vt_apply(const SView<T>& L, const T* v, const unsigned char* ex, int k) {
    T off = T(0);
    int cnt = 0;
    if (ex[k - 1]) off += v[k - 1], ++cnt;
    if (ex[k + 1]) off += v[k + 1], ++cnt;
    if (ex[k - vt::R]) off += v[k - vt::R], ++cnt;
    if (ex[k + vt::R]) off += v[k + vt::R], ++cnt;
    return L.c0 * (T(cnt) * v[k] - off);
}

template <typename T, typename TB>
__global__ void __launch_bounds__(kTileThreads)
    v_tile_down(SView<T> L, const TB* bin, const double* level_sum, T* bc, T* bp_out) {
    pdl_launch();
    constexpr int N = vt::R * vt::R;
    __shared__ T sb[N], sd[N], sx[N], sy[N], sr[N], ss[N];
    __shared__ unsigned char ex[N];
    __shared__ int nb9[9];
    const int b = blockIdx.x;
    vt_blocks(L, b, nb9);
    const bool project = L.singular && level_sum;
    const int4 mp = ld_static(reinterpret_cast<const int4*>(L.map + 4 * b));
    __syncthreads();
    // the region's loads, all issued before any is used; the volumes and
    // diagonals before the wait
    constexpr int QU = (N + kTileThreads - 1) / kTileThreads;
    int c[QU];
    TB a[QU];
    T vo[QU], dd[QU];
#pragma unroll
    for (int u = 0; u < QU; ++u) {
        const int q = threadIdx.x + u * kTileThreads;
        c[u] = q < N ? vt_cell(nb9, q % vt::R - 3, q / vt::R - 3) : -1;
    }
#pragma unroll
    for (int u = 0; u < QU; ++u) {
        if (c[u] >= 0) {
            vo[u] = (project && !L.const_vol) ? ld_static(L.vol + c[u]) : L.vol0;
            dd[u] = L.dinv ? ld_static(L.dinv + c[u]) : L.dinv0;
        }
    }
    pdl_wait();
    const double mean = project ? *level_sum * L.cvol_inv : 0.0;
#pragma unroll
    for (int u = 0; u < QU; ++u)
        if (c[u] >= 0) a[u] = bin[c[u]];
#pragma unroll
    for (int u = 0; u < QU; ++u) {
        const int q = threadIdx.x + u * kTileThreads;
        if (q >= N) continue;
        T bv = T(0), d = T(0);
        if (c[u] >= 0) {
            bv = mean != 0.0 ? T(double(a[u]) - double(vo[u]) * mean) : T(a[u]);
            d = dd[u];
        }
        ex[q] = c[u] >= 0;
        sb[q] = bv;
        sd[q] = d;
        sx[q] = L.w * d * bv;  // the first sweep from zero, pointwise
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 20 * 20; q += blockDim.x) {
        const int k = vt::at(q % 20 - 2, q / 20 - 2);
        if (ex[k]) sy[k] = sx[k] + L.w * sd[k] * (sb[k] - vt_apply(L, sx, ex, k));
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 18 * 18; q += blockDim.x) {
        const int k = vt::at(q % 18 - 1, q / 18 - 1);
        if (ex[k]) {
            const T r = sb[k] - vt_apply(L, sy, ex, k);
            sr[k] = r;
            ss[k] = sd[k] * r;
        }
    }
    __syncthreads();
    // t = r - wt A s on the block (into sx, no longer needed), and the block's
    // iterate (into L.y, read by v_tile_up) and projected right-hand side
    for (int q = threadIdx.x; q < 256; q += blockDim.x) {
        const int k = vt::at(q & 15, q >> 4);
        sx[k] = sr[k] - L.tw * vt_apply(L, ss, ex, k);
        L.y[b * 256 + q] = sy[k];
        if (bp_out) bp_out[b * 256 + q] = sb[k];
    }
    __syncthreads();
    if (mp.w == 1) {
        for (int q = threadIdx.x; q < 256; q += blockDim.x) {
            const int i = q & 15, j = q >> 4;
            const T t = sx[vt::at(i, j)];
            bc[mp.x * 256 + (mp.z + j) * 16 + mp.y + i] = t;
        }
    } else {
        // 2 x 2 aggregation in the order of v_restrict: row pairs, then the row above
        for (int q = threadIdx.x; q < 64; q += blockDim.x) {
            const int i = 2 * (q & 7), j = 2 * (q >> 3);
            const T h0 = sx[vt::at(i, j)] + sx[vt::at(i + 1, j)];
            const T d0 = sx[vt::at(i, j + 1)] + sx[vt::at(i + 1, j + 1)];
            const T t = h0 + d0;
            bc[mp.x * 256 + (mp.z + (j >> 1)) * 16 + mp.y + (i >> 1)] = t;
        }
    }
}

template <typename T, typename Epi>
__global__ void __launch_bounds__(kTileThreads)
    v_tile_up(SView<T> L, const T* xc, const T* bp_in, double* partial, unsigned* counter, double* mean_out, Epi epi) {
    pdl_launch();
    constexpr int N = vt::R * vt::R;
    __shared__ T se[N], sp[N], sq[N], sd[N], sb[N];
    __shared__ unsigned char ex[N];
    __shared__ int nb9[9];
    const int b = blockIdx.x;
    vt_blocks(L, b, nb9);
    __syncthreads();
    // the region's loads, all issued before any is used
    constexpr int QU = (N + kTileThreads - 1) / kTileThreads;
    int4 mp[QU];
    int c[QU], li[QU], lj[QU], ring[QU];
#pragma unroll
    for (int u = 0; u < QU; ++u) {
        const int q = threadIdx.x + u * kTileThreads;
        c[u] = -1;
        if (q < N) {
            const int i = q % vt::R - 3, j = q / vt::R - 3;
            const int bx = i < 0 ? -1 : (i > 15 ? 1 : 0), by = j < 0 ? -1 : (j > 15 ? 1 : 0);
            const int B = nb9[(by + 1) * 3 + bx + 1];
            li[u] = i - 16 * bx;
            lj[u] = j - 16 * by;
            // 3: the outer frame (e only), 2: x and D^-1 too, 1: also bp
            ring[u] = max(max(-i, i - 15), max(-j, j - 15));
            if (B >= 0) {
                c[u] = B * 256 + lj[u] * 16 + li[u];
                mp[u] = ld_static(reinterpret_cast<const int4*>(L.map + 4 * B));
            }
        }
    }
    T e[QU], x[QU], d[QU], bp[QU];
#pragma unroll
    for (int u = 0; u < QU; ++u) {
        e[u] = x[u] = d[u] = bp[u] = T(0);
        if (c[u] >= 0 && ring[u] <= 2) d[u] = L.dinv ? ld_static(L.dinv + c[u]) : L.dinv0;
    }
    pdl_wait();
#pragma unroll
    for (int u = 0; u < QU; ++u) {
        if (c[u] >= 0) {
            const int4 m = mp[u];
            e[u] = m.w == 1 ? xc[m.x * 256 + (m.z + lj[u]) * 16 + m.y + li[u]]
                            : xc[m.x * 256 + (m.z + (lj[u] >> 1)) * 16 + m.y + (li[u] >> 1)];
            if (ring[u] <= 2) {
                x[u] = L.y[c[u]];
                if (ring[u] <= 1) bp[u] = bp_in[c[u]];
            }
        }
    }
#pragma unroll
    for (int u = 0; u < QU; ++u) {
        const int q = threadIdx.x + u * kTileThreads;
        if (q >= N) continue;
        ex[q] = c[u] >= 0;
        se[q] = e[u];
        sp[q] = x[u];
        sd[q] = d[u];
        sb[q] = bp[u];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 20 * 20; q += blockDim.x) {
        const int k = vt::at(q % 20 - 2, q / 20 - 2);
        if (ex[k]) sp[k] += se[k] - L.tw * sd[k] * vt_apply(L, se, ex, k);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 18 * 18; q += blockDim.x) {
        const int k = vt::at(q % 18 - 1, q / 18 - 1);
        if (ex[k]) sq[k] = sp[k] + L.w * sd[k] * (sb[k] - vt_apply(L, sp, ex, k));
    }
    __syncthreads();
    double v = 0, w = 0;
    for (int q = threadIdx.x; q < 256; q += blockDim.x) {
        const int k = vt::at(q & 15, q >> 4);
        const T o = sq[k] + L.w * sd[k] * (sb[k] - vt_apply(L, sq, ex, k));
        const int c = b * 256 + q;
        L.x[c] = o;
        if (mean_out) {
            v += (L.const_vol ? double(L.vol0) : double(L.vol[c])) * double(o);
            if constexpr (Epi::kRz) w += double(epi.r[c]) * double(o);
        }
    }
    if (mean_out) fold_mean(v, w, partial, counter, mean_out, L.cvol_inv, epi);
}

}  // namespace tpa
