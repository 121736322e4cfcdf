// Kernels of the merged batch: many independent pressure solves (uneven tree
// depths) advanced together, one launch per V-cycle phase for every problem.
//
// Batch level j holds, for every problem k with L_k levels, its level
// l = j - (Lmax - L_k) when l >= 0 (levels aligned at the coarse end, so all
// coarsest levels share the last batch level).  Rows are concatenated in
// problem order; CSR columns, owners and child lists use batch-level row
// numbers.  Work is described by items of at most kItemRows rows that never
// straddle two problems (a work list per level), so a CTA's rows belong to one
// problem and per-problem sums fold per-item partials in item order
// (deterministic).  The smoother weight and the transfer weight are folded into
// per-row arrays wd = w D^-1 and td = wt Dt^-1 because they differ between
// problems.
//
// A level runs as two launches on the haloed block tiles of tiles.cuh (one tile
// list over all problems) or, when it is large, as six phases over its rows; the
// last level is one dense product per problem (bk_coarse).  What other kernels of
// the cycle write (`active`, states, vectors) comes through plain pointers: a
// const __restrict__ pointer marks its loads as invariant, and the compiler may
// then move them above the programmatic-launch wait.
#pragma once

#include <climits>
#include <cuda_runtime.h>

#include "cg_state.cuh"
#include "fused.cuh"
#include "solve_state.cuh"
#include "tiles.cuh"

namespace tpa {

constexpr int kItemRows = 256;
constexpr int kNoExt = INT_MIN;
// A batch level of at most this many tiles runs on them (two launches, one CTA's
// chain of loads and barriers per tile: 11 us at 211 tiles, 30 us at 529, 130 us
// at 3748); a larger one streams its rows through six phases, which execute a
// sixth of the tiles' instructions and are bound by the operator's bytes.
constexpr int kBatchTiles = 320;

// rows [begin, end) of problem `prob`; delta != kNoExt on a problem's finest
// level, where fine-space index = row + delta
struct BItem {
    int begin, end, prob, delta;
};

// A finest-level item of the CG (fine-space rows [begin, end); level row = row +
// off): kFineRows rows, each thread's kFinePer of them kItemRows apart, so that
// a fold (a fence and an atomic per item) is paid once per 1024 rows.
constexpr int kFinePer = 4;
constexpr int kFineRows = kFinePer * kItemRows;
struct BFItem {
    int begin, end, prob, lvl, off;
};

// The finest rows of every problem in FP64 (fine space): slices of 32 rows of an
// item, {first entry / 32, width}, entry u of row k at 32 u + k (columns are
// fine-space rows; padding holds 0 on the row itself), so that a warp's loads
// are consecutive.
struct FineRows {
    const int2* slice;
    const int* ci;
    const double* val;
    const double* vol;
};

// a problem's items, and the folds' scratch
struct FineFold {
    const int* first;
    const int* count;
    double* partial;
    int stride;
    unsigned* counters;
};

// One batch level: its vectors and, when its phases stream over the rows, the
// work items with the operator in slices of 32 rows of an item ({first entry / 32,
// width}, entry u of row k at 32 u + k; padding: value 0).  ci holds the columns,
// cc their owners (rows of the next coarser batch level).
template <typename T>
struct BLevel {
    const T* wd;   // w_k D^-1
    const T* td;   // wt_k Dt^-1
    const T* vol;
    const double* cvol_inv;     // per problem: 1 / component volume (0: no projection)
    T *b, *bp, *x, *y, *r;
    const BItem* items;
    const int2* slice;
    const T* val;
    const int* ci;
    const int* cc;
    const int* owner;
    // the coarse rows whose children lie in an item: co[cptr[item] ..), with the
    // item-local rows of their children (-1: none)
    const int* cptr;
    const int* co;
    const short4* ch;
    // where children straddle items (blocks wider than half an item): every coarse
    // row's problem and its children's rows
    const int* sprob;
    const int4* sch;
    int nsplit;                 // coarse rows of that form (0: by items)
    const int* pfirst;          // per problem: its first item (streamed) or tile
    const int* pcount;
    int nitems;
};

using BState = CgState;  // per-problem CG scalars

// N values folded over a problem's items [first, first + count); this CTA's item
// is blockIdx.x, value k at partial[k * stride + item]
template <int N, typename F>
__device__ __forceinline__ void fold_problem(const double (&v)[N], unsigned max_mask, double* partial, int stride,
                                             unsigned* counter, int first, int count, F done) {
    double* p[N];
    for (int k = 0; k < N; ++k) p[k] = partial + k * stride;
    fold_blocks<N>(v, max_mask, p, counter, blockIdx.x, first, count, done);
}

// ---- the tiled cycle ----------------------------------------------------------------

// a tile's problem, and on a problem's finest level its offset into fine space
// (kNoExt elsewhere)
struct BTile {
    int prob, delta;
};

// Right-hand side of a batch level's tiles: the level's own, or the fine-space
// residual projected by its sum on a problem's finest level.
template <typename T>
struct BTileRhs {
    const BTile* tiles;
    const double* cvol_inv;
    const double* ext;
    const T* b;
    const BState* st;
    const int* active;
    BTile t;
    double cv;
    __device__ __forceinline__ void prepare() {
        const int2 q = ld_static(reinterpret_cast<const int2*>(tiles + blockIdx.x));
        t = BTile{q.x, q.y};
        cv = ld_static(cvol_inv + t.prob);
    }
    __device__ __forceinline__ bool top() const { return t.delta != kNoExt; }
    __device__ __forceinline__ bool projects(const LevelView<T>&) const { return top() && cv != 0; }
    __device__ __forceinline__ bool start(const LevelView<T>& L, double& mean) const {
        mean = projects(L) ? st[t.prob].rsum * cv : 0.0;
        return active[t.prob] != 0;
    }
    __device__ __forceinline__ double load(int g) const { return top() ? ext[g + t.delta] : double(b[g]); }
};

template <typename T, int NT, int ROWS>
__global__ void __launch_bounds__(NT, 1)
    bk_tile_down(LevelView<T> L, TileView<T> V, BTileRhs<T> src, T* bc) {
    pdl_launch();
    src.prepare();
    tile_down<T, NT, ROWS>(with_weights(L), V, src, bc, src.top() ? L.bp : (T*)nullptr);
}

// gamma_next = r'z and the stopping rules of one problem (Krylov.jl `cg!`); init:
// the first one of a run.  One thread.
__device__ __forceinline__ void bk_after_z(BState* s, double g, int init, int* active) {
    bool stop;
    if (init) {
        s->gamma = g;
        s->pnorm2 = g;
        s->rnorm = sqrt(g);
        s->beta = 0;
        s->iter = 0;
        s->flags = g == 0 ? 8 : 0;
        stop = g == 0 || s->itmax <= 0;
    } else if (s->flags & 2) {
        stop = true;
    } else {
        const double rnorm = sqrt(g);
        s->rnorm = rnorm;
        const bool solved = rnorm + 1.0 <= 1.0;
        if (!solved) {
            const double beta = g / s->gamma;
            s->beta = beta;
            s->pnorm2 = g + beta * beta * s->pnorm2;
            s->gamma = g;
        } else {
            s->flags |= 4;
        }
        s->iter += 1;
        if (s->strong_max <= s->target) s->flags |= 1;
        stop = solved || s->iter >= s->itmax || (s->flags & 1);
    }
    if (stop) *active = 0;
}

// On a problem's finest level: the sums of V x and r x, which give the mean and
// r'z of z = x - mean.
template <typename T, int ROWS>
struct BTileOut {
    const T* vol;
    const double* r;
    const int* active;
    BTile t;
    T vv[ROWS];
    double rv[ROWS];
    double v = 0, w = 0;
    bool run = false;
    __device__ __forceinline__ void before(int q, int g, bool own) {
        if (t.delta != kNoExt && own) vv[q] = ld_static(vol + g);
    }
    __device__ __forceinline__ bool start() {
        run = active[t.prob] != 0;
        return run;
    }
    __device__ __forceinline__ void after(int q, int g, bool own) {
        if (t.delta != kNoExt && own) rv[q] = r[g + t.delta];
    }
    __device__ __forceinline__ void take(int q, double x) {
        if (t.delta == kNoExt) return;
        v += double(vv[q]) * x;
        w += rv[q] * x;
    }
};

template <typename T, int NT, int ROWS>
__global__ void __launch_bounds__(NT, 1)
    bk_tile_up(LevelView<T> L, TileView<T> V, const BTile* tiles, const double* cvol_inv, const T* xc, const double* r,
               const int* pfirst, const int* pcount, double* partial, int stride, unsigned* counters, double* mean_out, BState* st,
               int* active, int init) {
    pdl_launch();
    const int2 q = ld_static(reinterpret_cast<const int2*>(tiles + blockIdx.x));
    BTileOut<T, ROWS> out{L.vol, r, active, BTile{q.x, q.y}};
    tile_up<T, NT, ROWS>(with_weights(L), V, xc, (const T*)(q.y != kNoExt ? L.bp : L.b), out);
    if (!out.run || q.y == kNoExt) return;
    const double sums[2] = {out.v, out.w};
    fold_problem<2>(sums, 0u, partial, stride, counters + q.x, pfirst[q.x], pcount[q.x],
                    [&](const double (&t)[2]) {
                        const double mean = t[0] * cvol_inv[q.x];
                        mean_out[q.x] = mean;
                        bk_after_z(st + q.x, t[1] - mean * st[q.x].rsum, init, active + q.x);
                    });
}

// ---- the phases of a streamed level (one item per CTA) ------------------------------

__device__ __forceinline__ BItem batch_item(const BItem* items) {
    const int4 q = ld_static(reinterpret_cast<const int4*>(items + blockIdx.x));
    return BItem{q.x, q.y, q.z, q.w};
}

// A row of an item: its first kPre entries in registers, loaded before the wait;
// `col` is ci or cc.  Six entries hold a row away from refinement jumps and its
// right-hand side in 32 registers (FP32; 40 in FP64), every thread of an SM;
// eight take 40 and 48 and cost more in resident warps than they save at the
// jumps: 16 problems mixed 6.85 ms with eight, 6.54 with six; 256 problems 98 and
// 88 ms, FP64 126 and 111.
template <typename T>
struct BRow {
    static constexpr int kPre = 6;
    T a[kPre];
    int c[kPre];
    int w;
    const T* val;
    const int* col;
    __device__ __forceinline__ void load(const BLevel<T>& L, const int* cols) {
        const int2 s = ld_static(L.slice + size_t(blockIdx.x) * (kItemRows / 32) + (threadIdx.x >> 5));
        w = s.y;
        const size_t at = 32 * size_t(unsigned(s.x)) + (threadIdx.x & 31);
        val = L.val + at;
        col = cols + at;
#pragma unroll
        for (int u = 0; u < kPre; ++u)
            if (u < w) {
                a[u] = ld_static(val + 32 * u);
                c[u] = ld_static(col + 32 * u);
            }
    }
    // sum over the row, f(column) the vector's value
    template <typename F>
    __device__ __forceinline__ T dot(F f) const {
        T acc = T(0);
#pragma unroll
        for (int u = 0; u < kPre; ++u)
            if (u < w) acc += a[u] * f(c[u]);
        for (int u = kPre; u < w; ++u) acc += val[32 * u] * f(col[32 * u]);
        return acc;
    }
};

// both pre-sweeps from x = 0; on a problem's finest level the right-hand side is
// the fine-space residual `ext` (FP64), projected by its sum
template <typename T>
__global__ void __launch_bounds__(kItemRows) bk_pre2(BLevel<T> L, const double* ext, const BState* st,
                                                     const int* active) {
    pdl_launch();
    const BItem it = batch_item(L.items);
    BRow<T> row;
    row.load(L, L.ci);
    const int i = it.begin + int(threadIdx.x);
    const bool in = i < it.end;
    const T wd = in ? ld_static(L.wd + i) : T(0);
    pdl_wait();
    if (!active[it.prob] || !in) return;
    if (it.delta != kNoExt) {
        const double mean = st[it.prob].rsum * L.cvol_inv[it.prob];
        auto pb = [&](int q) { return T(ext[q + it.delta] - double(L.vol[q]) * mean); };
        const T bi = pb(i);
        const T acc = row.dot([&](int j) { return L.wd[j] * pb(j); });
        L.x[i] = wd * bi + wd * (bi - acc);
        L.bp[i] = bi;
    } else {
        const T bi = L.b[i];
        const T acc = row.dot([&](int j) { return L.wd[j] * L.b[j]; });
        L.x[i] = wd * bi + wd * (bi - acc);
    }
}

// r = bp - A x, s = td r (into y)
template <typename T>
__global__ void __launch_bounds__(kItemRows) bk_residual(BLevel<T> L, const int* active) {
    pdl_launch();
    const BItem it = batch_item(L.items);
    BRow<T> row;
    row.load(L, L.ci);
    const int i = it.begin + int(threadIdx.x);
    const bool in = i < it.end;
    const T td = in ? ld_static(L.td + i) : T(0);
    pdl_wait();
    if (!active[it.prob] || !in) return;
    const T* bp = it.delta != kNoExt ? L.bp : L.b;
    const T ri = bp[i] - row.dot([&](int j) { return L.x[j]; });
    L.r[i] = ri;
    L.y[i] = td * ri;
}

// b_c = P_tent'(r - A s): t per row in shared memory, then the item's coarse rows
// with their children in the fixed order (c0 + c1) + (c2 + c3); with straddling
// children (nsplit) t replaces r and bk_gather sums it
template <typename T>
__global__ void __launch_bounds__(kItemRows) bk_restrict(BLevel<T> L, T* bc, const int* active) {
    pdl_launch();
    __shared__ T t[kItemRows];
    const BItem it = batch_item(L.items);
    BRow<T> row;
    row.load(L, L.ci);
    const int i = it.begin + int(threadIdx.x);
    const bool split = L.nsplit > 0;
    const int J = split ? 0 : ld_static(L.cptr + blockIdx.x) + int(threadIdx.x);
    const int J1 = split ? 0 : ld_static(L.cptr + blockIdx.x + 1);
    short4 c = make_short4(-1, -1, -1, -1);
    int co = 0;
    if (J < J1) {
        c = ld_static(L.ch + J);
        co = ld_static(L.co + J);
    }
    pdl_wait();
    if (!active[it.prob]) return;
    if (i < it.end) {
        const T v = L.r[i] - row.dot([&](int j) { return L.y[j]; });
        if (split) L.r[i] = v;
        else t[threadIdx.x] = v;
    }
    __syncthreads();
    if (J >= J1) return;
    const T c0 = c.x >= 0 ? t[c.x] : T(0), c1 = c.y >= 0 ? t[c.y] : T(0);
    const T c2 = c.z >= 0 ? t[c.z] : T(0), c3 = c.w >= 0 ? t[c.w] : T(0);
    bc[co] = (c0 + c1) + (c2 + c3);
}

template <typename T>
__global__ void bk_gather(BLevel<T> L, T* bc, const int* active) {
    pdl_launch();
    const int J = blockIdx.x * blockDim.x + threadIdx.x;
    const int4 c = J < L.nsplit ? ld_static(L.sch + J) : make_int4(-1, -1, -1, -1);
    const int co = J < L.nsplit ? ld_static(L.co + J) : 0, prob = J < L.nsplit ? ld_static(L.sprob + J) : 0;
    pdl_wait();
    if (J >= L.nsplit || !active[prob]) return;
    const T c0 = c.x >= 0 ? L.r[c.x] : T(0), c1 = c.y >= 0 ? L.r[c.y] : T(0);
    const T c2 = c.z >= 0 ? L.r[c.z] : T(0), c3 = c.w >= 0 ? L.r[c.w] : T(0);
    bc[co] = (c0 + c1) + (c2 + c3);
}

// x += e - td A e, e = x_c(owner)
template <typename T>
__global__ void __launch_bounds__(kItemRows) bk_prolong(BLevel<T> L, const T* xc, const int* active) {
    pdl_launch();
    const BItem it = batch_item(L.items);
    BRow<T> row;
    row.load(L, L.cc);
    const int i = it.begin + int(threadIdx.x);
    const bool in = i < it.end;
    const T td = in ? ld_static(L.td + i) : T(0);
    const int o = in ? ld_static(L.owner + i) : 0;
    pdl_wait();
    if (!active[it.prob] || !in) return;
    L.x[i] += xc[o] - td * row.dot([&](int j) { return xc[j]; });
}

// a post-sweep out = in + wd (bp - A in); `fold`: on a problem's finest level the
// sums of V x and r x, which give the mean and r'z of z = x - mean
template <typename T, bool Fold>
__global__ void __launch_bounds__(kItemRows)
    bk_post(BLevel<T> L, const T* in_v, T* out_v, const double* ext, double* partial, int stride, unsigned* counters,
            double* mean_out, BState* st, int* active, int init) {
    pdl_launch();
    const BItem it = batch_item(L.items);
    BRow<T> row;
    row.load(L, L.ci);
    const int i = it.begin + int(threadIdx.x);
    const bool in = i < it.end, top = it.delta != kNoExt;
    const T wd = in ? ld_static(L.wd + i) : T(0);
    const double V = Fold && top && in ? double(ld_static(L.vol + i)) : 0.0;
    pdl_wait();
    if (!active[it.prob]) return;
    double sums[2] = {0, 0};
    if (in) {
        const T* bp = top ? L.bp : L.b;
        const T o = in_v[i] + wd * (bp[i] - row.dot([&](int j) { return in_v[j]; }));
        out_v[i] = o;
        if (Fold && top) {
            sums[0] = V * double(o);
            sums[1] = ext[i + it.delta] * double(o);
        }
    }
    if (!Fold || !top) return;
    fold_problem<2>(sums, 0u, partial, stride, counters + it.prob, L.pfirst[it.prob], L.pcount[it.prob],
                    [&](const double (&t)[2]) {
                        const double mean = t[0] * L.cvol_inv[it.prob];
                        mean_out[it.prob] = mean;
                        bk_after_z(st + it.prob, t[1] - mean * st[it.prob].rsum, init, active + it.prob);
                    });
}

// kCoarseRows rows of one problem's dense coarse solve (rows of the last level)
struct BCoarse {
    const double* G;
    int gn, begin, row, prob;
};
constexpr int kCoarseRows = 8;

// x = G b, a warp per row, the row's first 512 entries in flight before the
// wait.  G is the block of the augmented inverse: it sends the volumes to zero,
// so b needs no projection.
template <typename T>
__global__ void __launch_bounds__(32 * kCoarseRows)
    bk_coarse(const BCoarse* items, const T* b, T* x, const int* active) {
    pdl_launch();
    const BCoarse* p = items + blockIdx.x;
    const double* G = reinterpret_cast<const double*>(ld_static(reinterpret_cast<const long long*>(&p->G)));
    const int gn = ld_static(&p->gn), begin = ld_static(&p->begin), prob = ld_static(&p->prob);
    const int lane = threadIdx.x & 31, row = ld_static(&p->row) + int(threadIdx.x >> 5);
    if (row >= gn) {
        pdl_wait();
        return;
    }
    const double* g = G + size_t(row) * gn;
    double m[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) m[q] = lane + 32 * q < gn ? ld_static(g + lane + 32 * q) : 0.0;
    pdl_wait();
    if (!active[prob]) return;
    double acc = 0;
#pragma unroll
    for (int q = 0; q < 16; ++q)
        if (lane + 32 * q < gn) acc += m[q] * double(b[begin + lane + 32 * q]);
    for (int k = lane + 512; k < gn; k += 32) acc += g[k] * double(b[begin + k]);
    for (int o = 16; o; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (!lane) x[begin + row] = T(acc);
}

}  // namespace tpa
