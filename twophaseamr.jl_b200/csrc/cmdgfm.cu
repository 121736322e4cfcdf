// The CMDGFM two-block solve on the device (cmdgfm.cuh).
//
// ronaldremmerswaal/TwoPhaseAMR.jl solves the assembled system in
// `_project_cmdgfm_assembled!` (src/two_phase/projection/cmdgfm_projection.jl:
// 2201-2291): residual replacement around Krylov.jl 0.10 `bicgstab!` runs on
// the diagonally scaled system D_r M D_c (`_cmdgfm_krylov_scaling!`, :215-235)
// with the block preconditioner of :411-441 -- one V-cycle of the pressure
// hierarchy on the reduced pressure block (:374-405) and the incomplete LU of
// J - C D^-1 B on the jump block.  Here every vector lives in HBM, the
// V-cycle is the context's device cycle, the factor's triangular solves run
// level by level in one CTA with the vector in shared memory, and every
// reduction is a fixed-order fold of per-block partials (one block folds), so
// a solve repeats bit for bit.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "cmdgfm.cuh"
#include "fused.cuh"
#include "launch.cuh"

namespace tpa {
namespace {

constexpr int kT = 256;
constexpr int kG = 1184;  // 8 CTAs of 256 threads on each of 148 SMs
constexpr int kIluThreads = 1024;

inline int grid_of(int64_t n) {
    return int(std::max<int64_t>(1, std::min<int64_t>((n + kT - 1) / kT, kG)));
}

#define CM_LOOP(i, n) \
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < (n); i += int64_t(gridDim.x) * blockDim.x)

// state slots
enum : int {
    kRho = 0, kNextRho, kAlpha, kOmega, kBeta, kRnorm, kEps, kIter, kItmax, kFlags,
    kPressureDefect, kJumpDefect, kAnchorDefect, kRhsNorm2, kNonfinite, kChanged, kNorm2, kStateSize
};
enum : int { kSolved = 1, kTired = 2, kBreakdown = 4, kZeroRhs = 8, kZeroRho = 16 };

__device__ __forceinline__ double block_max_all(double v) {
    __shared__ double sh[32];
    for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (!lane) sh[wid] = v;
    __syncthreads();
    v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
    if (wid == 0)
        for (int o = 16; o; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// a NaN anywhere makes the maximum NaN
__device__ __forceinline__ double nan_max(double a, double b) { return (a != a || b != b) ? NAN : fmax(a, b); }

// ---------------------------------------------------------------- preconditioner

// The kernels of one BiCGSTAB iteration are short (3-10 us on the 25,000
// unknowns of a level-6 wave front) and each depends on the one before, so the
// iteration is bound by launches and load latencies, not by its bytes.  The
// iteration therefore has as few kernels as its reductions allow: dot products
// ride on the product that makes their operand, and the scalars they give are
// folded again by every CTA of the kernel that needs them (in the same order,
// so each CTA has the same value); one CTA stores them.  Each kernel is a
// programmatic dependent launch that loads its share of the system (pointers,
// columns, values, scales: written before the loop) and waits only then.  What
// the loop writes is read through plain pointers.  With 22 launches per
// iteration besides the V-cycles' own, a projection of that front took 4.51 ms;
// with these 11, 4.04 ms.

// full[cell_i] = src_i / rows_i (the reduced right-hand side scattered); with
// one component (anchor >= 0) the last block also writes full[anchor] = -(the
// sum of the values), folded from per-block partials in block order, and the
// sum of the whole, which is then zero unless a value is not finite
__global__ void k_cm_scatter(int64_t np, const double* src, const double* rows, const int32_t* cell, double* full,
                             int anchor, double* partial, unsigned* counter, double* total) {
    pdl_launch();
    const int64_t i0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    int32_t c0 = 0;
    double r0 = 1.0;
    if (i0 < np) {
        c0 = ld_static(cell + i0);
        r0 = ld_static(rows + i0);
    }
    pdl_wait();
    double v = 0;
    CM_LOOP(i, np) {
        const double q = src[i] / (i == i0 ? r0 : rows[i]);
        full[i == i0 ? c0 : cell[i]] = q;
        v += q;
    }
    if (anchor < 0) return;
    fold_sum(v, partial, counter, [&](double t) {
        full[anchor] = 0.0 - t;
        if (total) *total = t + (0.0 - t);
    });
}

// one block per anchor: full[anchor] = -(sum of its component's values)
__global__ void k_cm_anchor(const int32_t* gptr, const int32_t* gidx, const int32_t* ganchor, const double* src,
                            const double* rows, double* full) {
    pdl_entry();
    const int g = blockIdx.x;
    double v = 0;
    for (int k = gptr[g] + threadIdx.x; k < gptr[g + 1]; k += blockDim.x) {
        const int i = gidx[k];
        v += src[i] / rows[i];
    }
    v = block_sum_all(v);
    if (threadIdx.x == 0) full[ganchor[g]] = 0.0 - v;
}

// zp_i = z[cell_i] - z[anchor_i]; dst_i = zp_i / cols_i, z the V-cycle's result
// less its volume mean (read where the cycle left it: a pass that stores z
// first took 2.5 us and its launch)
template <typename T>
__global__ void k_cm_gather(int64_t np, const T* x, const double* mean, const int32_t* cell, const int32_t* anchor,
                            const double* cols, double* zp, double* dst) {
    pdl_launch();
    const int64_t i0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    int32_t c0 = 0, a0 = 0;
    double s0 = 1.0;
    if (i0 < np) {
        c0 = ld_static(cell + i0);
        a0 = ld_static(anchor + i0);
        s0 = ld_static(cols + i0);
    }
    pdl_wait();
    const double m = mean ? *mean : 0.0;
    CM_LOOP(i, np) {
        const bool first = i == i0;
        const double v = (double(x[first ? c0 : cell[i]]) - m) - (double(x[first ? a0 : anchor[i]]) - m);
        zp[i] = v;
        dst[i] = v / (first ? s0 : cols[i]);
    }
}

// One factor of the jump block laid out for its triangular solve: position i
// holds row rows[i], its entries (col, val)[ptr[i] .. ptr[i+1]) in column
// order and, for U, the reciprocal of its pivot inv[i].  `seq`: the positions
// are the rows in solve order (increasing for L, decreasing for U) and one
// thread walks them; otherwise the rows of level v are positions lev[v] ..
// lev[v+1], independent of each other, and the CTA takes each level between
// barriers.  A schedule whose levels hold few rows each -- the chains along
// the interface -- runs faster on one thread than with a barrier per level.

// copy a factor's arrays into shared memory at `at`; returns the view of the
// copy and advances `at` (8-byte aligned: doubles first)
template <bool Upper>
__device__ TriView stage(const TriView& g, int nx, char*& at) {
    TriView t = g;
    double* val = reinterpret_cast<double*>(at);
    double* inv = val + g.nnz;
    int32_t* lev = reinterpret_cast<int32_t*>(inv + (Upper ? nx : 0));
    int32_t* rows = lev + g.nlev + 1;
    int32_t* ptr = rows + nx;
    int32_t* col = ptr + nx + 1;
    for (int e = threadIdx.x; e < g.nnz; e += blockDim.x) {
        val[e] = g.val[e];
        col[e] = g.col[e];
    }
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
        rows[i] = g.rows[i];
        if (Upper) inv[i] = g.inv[i];
    }
    for (int i = threadIdx.x; i <= nx; i += blockDim.x) ptr[i] = g.ptr[i];
    for (int i = threadIdx.x; i <= g.nlev; i += blockDim.x) lev[i] = g.lev[i];
    t.val = val;
    t.inv = inv;
    t.lev = lev;
    t.rows = rows;
    t.ptr = ptr;
    t.col = col;
    at = reinterpret_cast<char*>(col + g.nnz);
    at += (8 - (reinterpret_cast<size_t>(at) & 7)) & 7;
    return t;
}

// The rows in solve order on one thread.  The next row's index, extent and
// first kPre entries are loaded into registers while the current row is
// summed, and the value just computed stays in a register for the next row,
// which in a chain along the interface usually needs it: the critical path
// per row is then one multiply-add and the reads of older values.
template <bool Upper>
__device__ __forceinline__ void walk_rows(double* __restrict__ y, const double* __restrict__ val,
                                          const double* __restrict__ inv, const int32_t* __restrict__ rows,
                                          const int32_t* __restrict__ ptr, const int32_t* __restrict__ col, int nx) {
    constexpr int kPre = 4;
    if (nx <= 0) return;
    int k = rows[0], e0 = ptr[0], e1 = ptr[1];
    int c[kPre];
    double v[kPre];
    for (int q = 0; q < kPre; ++q) {
        c[q] = e0 + q < e1 ? col[e0 + q] : 0;
        v[q] = e0 + q < e1 ? val[e0 + q] : 0.0;
    }
    double w = Upper ? inv[0] : 1.0;
    int klast = -1;
    double ylast = 0.0;
    for (int i = 0; i < nx; ++i) {
        const bool more = i + 1 < nx;
        const int nk = more ? rows[i + 1] : 0;
        const int ne1 = more ? ptr[i + 2] : e1;
        const double nw = (Upper && more) ? inv[i + 1] : 1.0;
        int nc[kPre];
        double nv[kPre];
        for (int q = 0; q < kPre; ++q) {
            nc[q] = e1 + q < ne1 ? col[e1 + q] : 0;
            nv[q] = e1 + q < ne1 ? val[e1 + q] : 0.0;
        }
        double acc = y[k];
        for (int q = 0; q < kPre; ++q)
            if (e0 + q < e1) {
                double yc;
                if (c[q] == klast) yc = ylast;
                else yc = y[c[q]];
                acc -= v[q] * yc;
            }
        for (int e = e0 + kPre; e < e1; ++e) acc -= val[e] * (col[e] == klast ? ylast : y[col[e]]);
        const double yk = Upper ? acc * w : acc;
        y[k] = yk;
        klast = k;
        ylast = yk;
        k = nk;
        e0 = e1;
        e1 = ne1;
        w = nw;
        for (int q = 0; q < kPre; ++q) {
            c[q] = nc[q];
            v[q] = nv[q];
        }
    }
}

template <bool Upper>
__device__ void tri_solve(const TriView& t, double* __restrict__ y, int nx) {
    auto row = [&](int i) {
        const int k = t.rows[i];
        double acc = y[k];
        for (int e = t.ptr[i]; e < t.ptr[i + 1]; ++e) acc -= t.val[e] * y[t.col[e]];
        y[k] = Upper ? acc * t.inv[i] : acc;
    };
    if (t.seq) {
        if (threadIdx.x == 0) walk_rows<Upper>(y, t.val, t.inv, t.rows, t.ptr, t.col, nx);
    } else {
        for (int v = 0; v < t.nlev; ++v) {
            for (int i = t.lev[v] + int(threadIdx.x); i < t.lev[v + 1]; i += blockDim.x) row(i);
            __syncthreads();
        }
    }
    __syncthreads();
}

// The jump block of the block preconditioner in one CTA: jr = src_xi / D_r -
// C zp, y = (L U)^-1 jr, dst_xi = y / D_c.  The vector lives in shared
// memory, and the factors too when `staged`.
__global__ void __launch_bounds__(kIluThreads)
    k_cm_jump_solve(int nx, int64_t np, const double* src, const double* rows, const int64_t* cptr,
                    const int32_t* ccol, const double* cval, const double* zp, TriView L, TriView U, int staged,
                    const double* cols, double* dst) {
    pdl_entry();
    extern __shared__ double sm[];
    double* y = sm;
    for (int f = threadIdx.x; f < nx; f += blockDim.x) {
        double acc = 0;
        for (int64_t e = cptr[f]; e < cptr[f + 1]; ++e) acc += cval[e] * zp[ccol[e]];
        y[f] = src[np + f] / rows[np + f] - acc;
    }
    if (staged) {
        char* at = reinterpret_cast<char*>(y + nx);
        L = stage<false>(L, nx, at);
        U = stage<true>(U, nx, at);
    }
    __syncthreads();
    if (staged && L.seq && U.seq) {
        // both factors walked on one thread, every array in shared memory
        if (threadIdx.x == 0) {
            const double* lval = reinterpret_cast<const double*>(y + nx);
            const int32_t* llev = reinterpret_cast<const int32_t*>(lval + L.nnz);
            const int32_t* lrows = llev + L.nlev + 1;
            const int32_t* lptr = lrows + nx;
            const int32_t* lcol = lptr + nx + 1;
            walk_rows<false>(y, lval, nullptr, lrows, lptr, lcol, nx);
            const char* at = reinterpret_cast<const char*>(lcol + L.nnz);
            at += (8 - (reinterpret_cast<size_t>(at) & 7)) & 7;
            const double* uval = reinterpret_cast<const double*>(at);
            const double* uinv = uval + U.nnz;
            const int32_t* ulev = reinterpret_cast<const int32_t*>(uinv + nx);
            const int32_t* urows = ulev + U.nlev + 1;
            const int32_t* uptr = urows + nx;
            const int32_t* ucol = uptr + nx + 1;
            walk_rows<true>(y, uval, uinv, urows, uptr, ucol, nx);
        }
        __syncthreads();
    } else {
        tri_solve<false>(L, y, nx);
        tri_solve<true>(U, y, nx);
    }
    for (int f = threadIdx.x; f < nx; f += blockDim.x) dst[np + f] = y[f] / cols[np + f];
}

// The jump block through the factors' inverses (triangular_inverses): jr =
// src_xi / D_r - C zp, y = L^-1 jr, x = U^-1 y, dst_xi = x / D_c, each a
// row-parallel product; one CTA, jr and y in shared memory.  Bound by the
// chain of loads along a row and from product to product, not by the 12,700
// entries of a level-6 wave front.  So a row is taken by as many lanes (`shift`:
// log2) as let one pass cover all rows, its bounds, its scales and the first
// entries of its C row are loaded before the wait, and so are both inverses,
// into shared memory, when they fit (`staged`).  By itself the kernel takes
// 9.9 us on that front (a thread per row with nothing loaded ahead: 9.7 us;
// eight lanes a row in four passes: 18.4 us), but its loads run beside the
// kernel before it: the solve's 46 products of this kind and all else on the
// device took 2.91 ms with it, 3.53 ms with the eight lanes.
__global__ void __launch_bounds__(kIluThreads)
    k_cm_jump_inverse(int nx, int64_t np, int shift, int staged, int lnnz, int unnz, const double* src,
                      const double* rows, const int64_t* cptr, const int32_t* ccol, const double* cval,
                      const double* zp, const int64_t* lptr, const int32_t* lcol, const double* lval,
                      const int64_t* uptr, const int32_t* ucol, const double* uval, const double* cols, double* dst) {
    constexpr int kHeld = 4;
    pdl_launch();
    extern __shared__ double sm[];
    double* a = sm;
    double* b = sm + nx;
    const int lanes = 1 << shift, lane = threadIdx.x & (lanes - 1);
    const int f0 = threadIdx.x >> shift;
    int64_t c0 = 0, c1 = 0, l0 = 0, l1 = 0, u0 = 0, u1 = 0;
    double scale_in = 1.0, scale_out = 1.0;
    if (f0 < nx) {
        c0 = ld_static(cptr + f0);
        c1 = ld_static(cptr + f0 + 1);
        l0 = ld_static(lptr + f0);
        l1 = ld_static(lptr + f0 + 1);
        u0 = ld_static(uptr + f0);
        u1 = ld_static(uptr + f0 + 1);
        scale_in = ld_static(rows + np + f0);
        scale_out = ld_static(cols + np + f0);
    }
    if (staged) {
        double* lv = b + nx;
        double* uv = lv + lnnz;
        int32_t* lc = reinterpret_cast<int32_t*>(uv + unnz);
        int32_t* uc = lc + lnnz;
#pragma unroll 4
        for (int e = threadIdx.x; e < lnnz; e += kIluThreads) {
            lv[e] = ld_static(lval + e);
            lc[e] = ld_static(lcol + e);
        }
#pragma unroll 4
        for (int e = threadIdx.x; e < unnz; e += kIluThreads) {
            uv[e] = ld_static(uval + e);
            uc[e] = ld_static(ucol + e);
        }
        lval = lv;
        lcol = lc;
        uval = uv;
        ucol = uc;
    }
    int32_t hc[kHeld];
    double hv[kHeld];
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
        const int64_t e = c0 + lane + (k << shift);
        hc[k] = e < c1 ? ld_static(ccol + e) : 0;
        hv[k] = e < c1 ? ld_static(cval + e) : 0.0;
    }
    pdl_wait();
    // this lane's part of a row, kHeld entries in flight; summed over the row's lanes
    auto along = [&](int64_t e0, int64_t e1, const int32_t* col, const double* val, const double* v) {
        double acc = 0;
        for (int64_t e = e0 + lane; e < e1; e += int64_t(kHeld) << shift) {
            double t[kHeld];
#pragma unroll
            for (int k = 0; k < kHeld; ++k) {
                const int64_t q = e + (k << shift);
                t[k] = q < e1 ? val[q] * v[col[q]] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < kHeld; ++k) acc += t[k];
        }
        return acc;
    };
    // every lane of a warp takes the same trips, so that the shuffles see all of them
    auto total = [&](double acc) {
        for (int o = lanes >> 1; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        return acc;
    };
    const int step = kIluThreads >> shift;
    for (int base = 0; base < nx; base += step) {
        const int f = base + f0;
        double acc = 0;
        if (base == 0) {
#pragma unroll
            for (int k = 0; k < kHeld; ++k)
                if (c0 + lane + (k << shift) < c1) acc += hv[k] * zp[hc[k]];
            acc += along(c0 + (int64_t(kHeld) << shift), c1, ccol, cval, zp);
        } else if (f < nx) {
            acc = along(cptr[f], cptr[f + 1], ccol, cval, zp);
        }
        acc = total(acc);
        if (f < nx && lane == 0) a[f] = src[np + f] / (base ? rows[np + f] : scale_in) - acc;
    }
    __syncthreads();
    for (int base = 0; base < nx; base += step) {
        const int f = base + f0;
        double acc = 0;
        if (f < nx) acc = along(base ? lptr[f] : l0, base ? lptr[f + 1] : l1, lcol, lval, a);
        acc = total(acc);
        if (f < nx && lane == 0) b[f] = acc;
    }
    __syncthreads();
    for (int base = 0; base < nx; base += step) {
        const int f = base + f0;
        double acc = 0;
        if (f < nx) acc = along(base ? uptr[f] : u0, base ? uptr[f + 1] : u1, ucol, uval, b);
        acc = total(acc);
        if (f < nx && lane == 0) dst[np + f] = acc / (base ? cols[np + f] : scale_out);
    }
}

// ---------------------------------------------------------------- products

// y = A x with A = D_r M D_c, and with it the block partials of c'y (p1) and,
// with `yy`, of y'y (p2): a row per thread, whose pointers, scale and first
// kHeld entries -- the whole row of a cell away from the front -- are loaded
// before the wait, so that only x is read after it
__global__ void __launch_bounds__(kT)
    k_cm_product(int64_t n, const int64_t* ptr, const int32_t* col, const double* val, const double* rows,
                 const double* cols, const double* x, double* y, const double* c, int yy, double* p1, double* p2) {
    constexpr int kHeld = 6;
    pdl_launch();
    int32_t hc[kHeld];
    double hv[kHeld], hs[kHeld];
    int64_t e0 = 0, e1 = 0;
    double scale = 0;
    const int64_t i0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i0 < n) {
        e0 = ld_static(ptr + i0);
        e1 = ld_static(ptr + i0 + 1);
        scale = ld_static(rows + i0);
    }
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
        const bool in = e0 + k < e1;
        hc[k] = in ? ld_static(col + e0 + k) : 0;
        hv[k] = in ? ld_static(val + e0 + k) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kHeld; ++k) hs[k] = e0 + k < e1 ? ld_static(cols + hc[k]) : 0.0;
    pdl_wait();
    double v = 0, w = 0;
    auto put = [&](int64_t i, double yi) {
        y[i] = yi;
        v += c[i] * yi;
        if (yy) w += yi * yi;
    };
    if (i0 < n) {
        double acc = 0;
#pragma unroll
        for (int k = 0; k < kHeld; ++k)
            if (e0 + k < e1) acc += hv[k] * (hs[k] * x[hc[k]]);
        for (int64_t e = e0 + kHeld; e < e1; ++e) acc += val[e] * (cols[col[e]] * x[col[e]]);
        put(i0, scale * acc);
    }
    for (int64_t i = i0 + int64_t(gridDim.x) * blockDim.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        double acc = 0;
        for (int64_t e = ptr[i]; e < ptr[i + 1]; ++e) acc += val[e] * (cols[col[e]] * x[col[e]]);
        put(i, rows[i] * acc);
    }
    v = block_sum_all(v);
    if (yy) w = block_sum_all(w);
    if (threadIdx.x == 0) {
        p1[blockIdx.x] = v;
        if (yy) p2[blockIdx.x] = w;
    }
}

// corr = rhs - M sol
__global__ void k_cm_residual(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ col,
                              const double* __restrict__ val, const double* __restrict__ rhs,
                              const double* __restrict__ sol, double* __restrict__ corr) {
    CM_LOOP(i, n) {
        double acc = 0;
        for (int64_t e = ptr[i]; e < ptr[i + 1]; ++e) acc += val[e] * sol[col[e]];
        corr[i] = rhs[i] - acc;
    }
}

// block partials of a'a
__global__ void k_cm_norm2(int64_t n, const double* __restrict__ a, double* __restrict__ p1) {
    double v = 0;
    CM_LOOP(i, n) v += a[i] * a[i];
    v = block_sum_all(v);
    if (threadIdx.x == 0) p1[blockIdx.x] = v;
}

// ---------------------------------------------------------------- BiCGSTAB

// x = 0, r = p = b, v = 0, with the partials of r'r (= c'r: the shadow
// residual c is b itself)
__global__ void k_cm_init(int64_t n, const double* __restrict__ b, double* __restrict__ x, double* __restrict__ r,
                          double* __restrict__ p, double* __restrict__ v, double* __restrict__ p1) {
    double w = 0;
    CM_LOOP(i, n) {
        const double bi = b[i];
        x[i] = 0.0;
        r[i] = bi;
        p[i] = bi;
        v[i] = 0.0;
        w += bi * bi;
    }
    w = block_sum_all(w);
    if (threadIdx.x == 0) p1[blockIdx.x] = w;
}

// rNorm, eps = atol + rtol rNorm, rho_1 = c'r (= rNorm^2: c = r = b)
__global__ void k_cm_init_fold(const double* p1, int count, double rtol, int itmax, double* st) {
    const double rr = fold_partials(p1, count);
    if (threadIdx.x == 0) {
        const double rnorm = sqrt(rr);
        st[kRnorm] = rnorm;
        st[kEps] = 0.0 + rtol * rnorm;
        st[kNextRho] = rr;
        st[kIter] = 0;
        st[kItmax] = itmax;
        int flags = 0;
        if (rnorm == 0.0) flags |= kZeroRhs;
        else if (rr == 0.0) flags |= kZeroRho;
        if (rnorm <= st[kEps]) flags |= kSolved;
        if (itmax <= 0) flags |= kTired;
        st[kFlags] = flags;
    }
}

// a fold's value, which thread 0 holds, handed to every thread of the CTA
__device__ __forceinline__ double to_all(double v) {
    __shared__ double one;
    __syncthreads();
    if (threadIdx.x == 0) one = v;
    __syncthreads();
    return one;
}

// rho = next_rho; alpha = rho / c'v (from the partials p1)
// s = r - alpha v; x = x + alpha y
__global__ void k_cm_update1(int64_t n, const double* p1, int count, const double* r, const double* v,
                             const double* y, double* s, double* x, double* st) {
    pdl_entry();
    const double rho = st[kNextRho];
    const double a = rho / to_all(fold_partials(p1, count));
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st[kRho] = rho;
        st[kAlpha] = a;
    }
    CM_LOOP(i, n) {
        s[i] = r[i] - a * v[i];
        x[i] = x[i] + a * y[i];
    }
}

// omega = t's / t't (from the partials p1, p2)
// x = x + omega z; r = s - omega t; partials of c'r (p3) and r'r (p4)
__global__ void k_cm_update2(int64_t n, const double* p1, const double* p2, int count, const double* s,
                             const double* t, const double* z, const double* c, double* x, double* r, double* st,
                             double* p3, double* p4) {
    pdl_entry();
    const double ts = fold_partials(p1, count);
    const double tt = fold_partials(p2, count);
    const double w = to_all(ts / tt);
    if (blockIdx.x == 0 && threadIdx.x == 0) st[kOmega] = w;
    double cr = 0, rr = 0;
    CM_LOOP(i, n) {
        x[i] = x[i] + w * z[i];
        const double ri = s[i] - w * t[i];
        r[i] = ri;
        cr += c[i] * ri;
        rr += ri * ri;
    }
    cr = block_sum_all(cr);
    rr = block_sum_all(rr);
    if (threadIdx.x == 0) {
        p3[blockIdx.x] = cr;
        p4[blockIdx.x] = rr;
    }
}

// next_rho, beta, rNorm and the stopping rules of the iteration (from the
// partials p3, p4), which one CTA stores; p = r + beta (p - omega v)
__global__ void k_cm_pupdate(int64_t n, const double* p3, const double* p4, int count, const double* r,
                             const double* v, double* p, double* st, cudaGraphConditionalHandle handle,
                             int set_cond) {
    pdl_entry();
    const double a = st[kAlpha], w = st[kOmega];
    const double cr = to_all(fold_partials(p3, count));
    const double b = (cr / st[kRho]) * (a / w);
    CM_LOOP(i, n) p[i] = r[i] + b * (p[i] - w * v[i]);
    if (blockIdx.x != 0) return;
    const double rr = fold_partials(p4, count);
    if (threadIdx.x == 0) {
        st[kNextRho] = cr;
        st[kBeta] = b;
        const double rnorm = sqrt(rr);
        st[kRnorm] = rnorm;
        const double iter = st[kIter] + 1;
        st[kIter] = iter;
        int flags = 0;
        if (rnorm <= st[kEps] || rnorm + 1.0 <= 1.0) flags |= kSolved;
        if (iter >= st[kItmax]) flags |= kTired;
        if (a == 0.0 || a != a) flags |= kBreakdown;
        st[kFlags] = flags;
        if (set_cond) cudaGraphSetConditional(handle, (flags & (kSolved | kTired | kBreakdown)) ? 0u : 1u);
    }
}

// ---------------------------------------------------------------- residual replacement

// block partials: max weighted |corr| over pressure rows (p1), over jump rows
// (p2), and sum (rows corr)^2 (p3)
__global__ void k_cm_defects(int64_t n, int64_t np, const double* __restrict__ corr,
                             const double* __restrict__ weight, const double* __restrict__ rows, double* __restrict__ p1,
                             double* __restrict__ p2, double* __restrict__ p3) {
    double mp = 0, mj = 0, s2 = 0;
    CM_LOOP(i, n) {
        const double d = weight[i] * fabs(corr[i]);
        if (i < np) mp = nan_max(mp, d);
        else mj = nan_max(mj, d);
        const double q = rows[i] * corr[i];
        s2 += q * q;
    }
    bool nanp = mp != mp, nanj = mj != mj;
    mp = block_max_all(nanp ? 0.0 : mp);
    mj = block_max_all(nanj ? 0.0 : mj);
    s2 = block_sum_all(s2);
    __shared__ int any[2];
    if (threadIdx.x == 0) any[0] = any[1] = 0;
    __syncthreads();
    if (nanp) any[0] = 1;
    if (nanj) any[1] = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        p1[blockIdx.x] = any[0] ? NAN : mp;
        p2[blockIdx.x] = any[1] ? NAN : mj;
        p3[blockIdx.x] = s2;
    }
}

// the omitted anchor rows at the current solution: block maxima of
// weight_a |rhs_a - (E sol)_a|
__global__ void k_cm_anchor_defect(int64_t na, const int64_t* __restrict__ ptr, const int32_t* __restrict__ col,
                                   const double* __restrict__ val, const double* __restrict__ rhs,
                                   const double* __restrict__ w, const double* __restrict__ sol,
                                   double* __restrict__ p4) {
    double m = 0;
    bool nan = false;
    CM_LOOP(a, na) {
        double acc = 0;
        for (int64_t e = ptr[a]; e < ptr[a + 1]; ++e) acc += val[e] * sol[col[e]];
        const double d = w[a] * fabs(rhs[a] - acc);
        if (d != d) nan = true;
        else m = fmax(m, d);
    }
    __shared__ int any;
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    if (nan) any = 1;
    m = block_max_all(m);
    if (threadIdx.x == 0) p4[blockIdx.x] = any ? NAN : m;
}

__device__ double fold_max(const double* p, int count) {
    double m = 0;
    bool nan = false;
    for (int k = threadIdx.x; k < count; k += blockDim.x) {
        const double v = ((volatile const double*)p)[k];
        if (v != v) nan = true;
        else m = fmax(m, v);
    }
    __shared__ int any;
    __syncthreads();  // a previous call's readers of `any` are done
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    if (nan) any = 1;
    m = block_max_all(m);
    __syncthreads();
    return any ? NAN : m;
}

__global__ void k_cm_defects_fold(const double* p1, const double* p2, const double* p3, int count,
                                  const double* p4, int count4, double* st) {
    const double mp = fold_max(p1, count);
    const double mj = fold_max(p2, count);
    const double s2 = fold_partials(p3, count);
    const double ma = count4 > 0 ? fold_max(p4, count4) : 0.0;
    if (threadIdx.x == 0) {
        st[kPressureDefect] = mp;
        st[kJumpDefect] = mj;
        st[kRhsNorm2] = s2;
        st[kAnchorDefect] = ma;
    }
}

// b = rows corr, divided by `norm` when normalize
__global__ void k_cm_scaled_rhs(int64_t n, const double* __restrict__ rows, const double* __restrict__ corr,
                                double* __restrict__ b, int normalize, double norm) {
    CM_LOOP(i, n) {
        const double v = rows[i] * corr[i];
        b[i] = normalize ? v / norm : v;
    }
}

// block partials: non-finite entries of x (p1)
__global__ void k_cm_nonfinite(int64_t n, const double* __restrict__ x, double* __restrict__ p1) {
    double c = 0;
    CM_LOOP(i, n) if (!isfinite(x[i])) c += 1.0;
    c = block_sum_all(c);
    if (threadIdx.x == 0) p1[blockIdx.x] = c;
}

// sol = sol + cols (scale x), block partials of the changed entries (p1)
__global__ void k_cm_apply(int64_t n, double* __restrict__ sol, const double* __restrict__ cols, double scale,
                           const double* __restrict__ x, double* __restrict__ p1) {
    double c = 0;
    CM_LOOP(i, n) {
        const double prev = sol[i];
        const double upd = prev + cols[i] * (scale * x[i]);
        sol[i] = upd;
        if (upd != prev) c += 1.0;
    }
    c = block_sum_all(c);
    if (threadIdx.x == 0) p1[blockIdx.x] = c;
}

__global__ void k_cm_sum_fold(const double* p1, int count, double* out) {
    const double v = fold_partials(p1, count);
    if (threadIdx.x == 0) *out = v;
}

}  // namespace

// ---------------------------------------------------------------- host driver

// dst = (N^-1 (src / D_r)) / D_c: `_ScaledProjectionPreconditioner` around
// the block preconditioner (cmdgfm_projection.jl:158-179, 374-441)
void CmdgfmDevice::precondition(DeviceSolver& ds, const double* src, double* dst, int precision, cudaStream_t s) {
    const Launch go{s, ds.pdl()};
    if (np_ > 0) {
        // one component: the anchor's value folds in the scatter, and with it the
        // cycle's right-hand-side sum; several: one block each, and a pass for the sum
        const bool one = ngroups_ == 1;
        go(k_cm_scatter, grid_of(np_), kT, 0, np_, src, rows_.p, cell_.p, full_.p, one ? anchor1_ : -1,
           partial_.p + 2 * kG, counter_.p, ds.fused() ? ds.cycle_rhs_sum() : nullptr);
        ++launches_;
        if (ngroups_ > 1) {
            go(k_cm_anchor, ngroups_, 1024, 0, gptr_.p, gidx_.p, ganchor_.p, src, rows_.p, full_.p);
            ++launches_;
        }
        const int before = ds.kernel_launches();
        if (ds.fused()) {
            const DeviceSolver::CycleResult z = ds.vcycle_result(full_.p, precision, one);
            if (precision)
                go(k_cm_gather<float>, grid_of(np_), kT, 0, np_, z.xf, z.mean, cell_.p, anchor_.p, cols_.p, zp_.p, dst);
            else
                go(k_cm_gather<double>, grid_of(np_), kT, 0, np_, z.xd, z.mean, cell_.p, anchor_.p, cols_.p, zp_.p,
                   dst);
        } else {
            ds.vcycle(full_.p, zfull_.p, precision);
            go(k_cm_gather<double>, grid_of(np_), kT, 0, np_, zfull_.p, nullptr, cell_.p, anchor_.p, cols_.p, zp_.p,
               dst);
        }
        launches_ += ds.kernel_launches() - before + 1;
    }
    if (nx_ > 0) jump_apply(ds, src, rows_.p, cols_.p, zp_.p, dst, s);
}

// One BiCGSTAB iteration (Krylov.jl 0.10 `bicgstab!` with the right
// preconditioner N): y = N^-1 p, v = A y, alpha; s = r - alpha v, x += alpha y;
// z = N^-1 s, t = A z, omega; x += omega z, r = s - omega t; next rho, beta,
// rNorm and the stopping rules (which set the loop condition when `set_cond`);
// p = r + beta (p - omega v).
void CmdgfmDevice::enqueue_iteration(DeviceSolver& ds, bool preconditioned, int precision, cudaStream_t s,
                                     cudaGraphConditionalHandle handle, int set_cond) {
    const Launch go{s, ds.pdl()};
    const int g = grid_of(n_);
    double* const pt = partial_.p;
    double* st = state_.p;
    // w = A u with the partials of c'w (and w'w)
    auto product = [&](const double* u, double* w, const double* c, int ww) {
        go(k_cm_product, g, kT, 0, n_, mptr_.p, mcol_.p, mval_.p, rows_.p, cols_.p, u, w, c, ww, pt, pt + kG);
    };
    const double* y = p_.p;
    if (preconditioned) {
        precondition(ds, p_.p, y_.p, precision, s);
        y = y_.p;
    }
    product(y, v_.p, c_.p, 0);
    go(k_cm_update1, g, kT, 0, n_, pt, g, r_.p, v_.p, y, s_.p, x_.p, st);
    const double* z = s_.p;
    if (preconditioned) {
        precondition(ds, s_.p, z_.p, precision, s);
        z = z_.p;
    }
    product(z, t_.p, s_.p, 1);
    go(k_cm_update2, g, kT, 0, n_, pt, pt + kG, g, s_.p, t_.p, z, c_.p, x_.p, r_.p, st, pt + 2 * kG, pt + 3 * kG);
    go(k_cm_pupdate, g, kT, 0, n_, pt + 2 * kG, pt + 3 * kG, g, r_.p, v_.p, p_.p, st, handle, set_cond);
    launches_ += 5;
}

// The iteration captured as the body of a graph WHILE node, kept while every
// argument it captured is unchanged: the sizes, the jump-block layout, the
// buffers and the pressure hierarchy's graph generation.
cudaGraphExec_t CmdgfmDevice::loop_graph(DeviceSolver& ds, bool preconditioned, int precision, cudaStream_t s) {
    std::vector<uintptr_t> key = {
        uintptr_t(n_), uintptr_t(np_), uintptr_t(nx_), uintptr_t(ncells_), uintptr_t(ngroups_),
        uintptr_t(int64_t(anchor1_)), uintptr_t(precision), uintptr_t(inverse_), uintptr_t(jstaged_),
        uintptr_t(jsmem_), uintptr_t(inverse_ ? ismem_ : 0), uintptr_t(inverse_ ? linnz_ : 0),
        uintptr_t(inverse_ ? uinnz_ : 0), uintptr_t(ds.graph_generation()), uintptr_t(s)};
    for (const void* q : {(const void*)mptr_.p, (const void*)mcol_.p, (const void*)mval_.p, (const void*)rows_.p,
                          (const void*)cols_.p, (const void*)cell_.p, (const void*)anchor_.p, (const void*)gptr_.p,
                          (const void*)gidx_.p, (const void*)ganchor_.p, (const void*)cptr_.p, (const void*)ccol_.p,
                          (const void*)cval_.p, (const void*)liptr_.p, (const void*)licol_.p, (const void*)lival_.p,
                          (const void*)uiptr_.p, (const void*)uicol_.p, (const void*)uival_.p, (const void*)x_.p,
                          (const void*)r_.p, (const void*)c_.p, (const void*)p_.p, (const void*)v_.p,
                          (const void*)s_.p, (const void*)t_.p, (const void*)y_.p, (const void*)z_.p,
                          (const void*)full_.p, (const void*)zfull_.p, (const void*)zp_.p, (const void*)partial_.p,
                          (const void*)state_.p, (const void*)counter_.p})
        key.push_back(reinterpret_cast<uintptr_t>(q));
    for (const TriView* v : {&lview_, &uview_}) {
        const unsigned char* b = reinterpret_cast<const unsigned char*>(v);
        for (size_t i = 0; i < sizeof(TriView); i += sizeof(uintptr_t)) {
            uintptr_t w = 0;
            std::memcpy(&w, b + i, std::min(sizeof(uintptr_t), sizeof(TriView) - i));
            key.push_back(w);
        }
    }
    const int slot = preconditioned ? 1 : 0;
    if (exec_[slot] && key == key_[slot]) return exec_[slot];
    if (exec_[slot]) cudaGraphExecDestroy(exec_[slot]);
    exec_[slot] = nullptr;
    cudaGraph_t graph;
    TPA_CUDA(cudaGraphCreate(&graph, 0));
    cudaGraphConditionalHandle handle;
    TPA_CUDA(cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault));
    alignas(cudaGraphNodeParams) unsigned char cp_storage[sizeof(cudaGraphNodeParams)];
    std::memset(cp_storage, 0, sizeof(cp_storage));
    cudaGraphNodeParams& cp = *reinterpret_cast<cudaGraphNodeParams*>(cp_storage);
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    TPA_CUDA(cudaGraphAddNode(&node, graph, nullptr, 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    const int before = launches_, ds_before = ds.kernel_launches();
    TPA_CUDA(cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    enqueue_iteration(ds, preconditioned, precision, s, handle, 1);
    cudaGraph_t captured;
    const cudaError_t ce = cudaStreamEndCapture(s, &captured);
    body_launches_[slot] = (launches_ - before);
    launches_ = before;
    ds.add_launches(ds_before - ds.kernel_launches());  // the capture launched nothing
    if (ce != cudaSuccess) {
        cudaGraphDestroy(graph);
        throw Error(2, std::string("graph capture failed: ") + cudaGetErrorString(ce));
    }
    cudaGraphExec_t exec;
    const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) throw Error(2, std::string("graph instantiation failed: ") + cudaGetErrorString(ie));
    exec_[slot] = exec;
    key_[slot] = key;
    return exec;
}

// dst_xi = (L U)^-1 (src_xi / rows_xi - C zp) / cols_xi: the jump block of the
// block preconditioner (rows, cols: D_r, D_c) or of the warm start (ones)
void CmdgfmDevice::jump_apply(DeviceSolver& ds, const double* src, const double* rows, const double* cols,
                              const double* zp, double* dst, cudaStream_t s) {
    const Launch go{s, ds.pdl()};
    if (inverse_)
        go(k_cm_jump_inverse, 1, kIluThreads, ismem_, int(nx_), np_, ishift_, istaged_, linnz_, uinnz_, src, rows,
           cptr_.p, ccol_.p, cval_.p, zp, liptr_.p, licol_.p, lival_.p, uiptr_.p, uicol_.p, uival_.p, cols, dst);
    else
        go(k_cm_jump_solve, 1, kIluThreads, jsmem_, int(nx_), np_, src, rows, cptr_.p, ccol_.p, cval_.p, zp, lview_,
           uview_, jstaged_, cols, dst);
    ++launches_;
}

int CmdgfmDevice::bicgstab(DeviceSolver& ds, const CmdgfmInput& in, const CmdgfmFactor& f, bool preconditioned,
                           double rtol, int itmax, cudaStream_t s) {
    const int g = grid_of(n_);
    double* p1 = partial_.p;
    double* st = state_.p;
    double hs[kStateSize];
    auto read = [&] {
        TPA_CUDA(cudaMemcpyAsync(hs, st, sizeof(hs), cudaMemcpyDeviceToHost, s));
        TPA_CUDA(cudaStreamSynchronize(s));
    };
    // x0 = 0, r = p = b (= c_), the shadow residual c = b
    k_cm_init<<<g, kT, 0, s>>>(n_, c_.p, x_.p, r_.p, p_.p, v_.p, p1);
    k_cm_init_fold<<<1, kT, 0, s>>>(p1, g, rtol, itmax, st);
    launches_ += 2;
    read();
    if (int(hs[kFlags]) & (kZeroRhs | kZeroRho | kSolved | kTired)) return 0;
    if (s && !std::getenv("TPAGMG_NO_GRAPH")) {
        // the whole run as one graph launch; the host reads the state at its end
        cudaGraphExec_t exec = loop_graph(ds, preconditioned, in.precision, s);
        TPA_CUDA(cudaGraphLaunch(exec, s));
        read();
        launches_ += int(hs[kIter]) * body_launches_[preconditioned ? 1 : 0];
    } else {
        for (;;) {
            enqueue_iteration(ds, preconditioned, in.precision, s, cudaGraphConditionalHandle(), 0);
            read();
            if (int(hs[kFlags]) & (kSolved | kTired | kBreakdown)) break;
        }
    }
    TPA_CUDA(cudaGetLastError());
    return int(hs[kIter]);
}

void CmdgfmDevice::solve(DeviceSolver& ds, const CmdgfmInput& in, const CmdgfmFactor& f, double* solution,
                         CmdgfmStats& st) {
    const double eps = 2.220446049250313e-16;
    cudaStream_t s = ds.stream();
    st = CmdgfmStats();
    n_ = in.m.n;
    np_ = in.np;
    nx_ = n_ - np_;
    na_ = in.extra.n;
    ncells_ = ds.ncells();
    launches_ = 0;
    if (nx_ * int64_t(sizeof(double)) > 200 * 1024)
        throw Error(5, "the jump block has more than 25,600 unknowns (its factor solve keeps them in shared memory)");
    cudaEvent_t e0, e1;
    TPA_CUDA(cudaEventCreate(&e0));
    TPA_CUDA(cudaEventCreate(&e1));
    TPA_CUDA(cudaEventRecord(e0, s));
    // the system and the factor
    mptr_.upload(in.m.ptr.data(), in.m.ptr.size(), s);
    mcol_.upload(in.m.col.data(), in.m.col.size(), s);
    mval_.upload(in.m.val.data(), in.m.val.size(), s);
    rhs_.upload(in.rhs.data(), in.rhs.size(), s);
    weight_.upload(in.weight.data(), in.weight.size(), s);
    rows_.upload(in.row_scale.data(), in.row_scale.size(), s);
    cols_.upload(in.col_scale.data(), in.col_scale.size(), s);
    cell_.upload(in.cell.data(), in.cell.size(), s);
    anchor_.upload(in.anchor.data(), in.anchor.size(), s);
    eptr_.upload(in.extra.ptr.data(), in.extra.ptr.size(), s);
    ecol_.upload(in.extra.col.data(), in.extra.col.size(), s);
    eval_.upload(in.extra.val.data(), in.extra.val.size(), s);
    erhs_.upload(in.extra_rhs.data(), in.extra_rhs.size(), s);
    eweight_.upload(in.extra_weight.data(), in.extra_weight.size(), s);
    // anchors and their members (indices increasing) for the reduced scatter
    std::vector<int32_t> anchors(in.anchor.begin(), in.anchor.end());
    std::sort(anchors.begin(), anchors.end());
    anchors.erase(std::unique(anchors.begin(), anchors.end()), anchors.end());
    ngroups_ = int(anchors.size());
    std::vector<int32_t> gptr(static_cast<size_t>(ngroups_) + 1, 0), gidx(static_cast<size_t>(np_));
    for (int64_t i = 0; i < np_; ++i) {
        const int g = int(std::lower_bound(anchors.begin(), anchors.end(), in.anchor[size_t(i)]) - anchors.begin());
        ++gptr[size_t(g) + 1];
    }
    for (int g = 0; g < ngroups_; ++g) gptr[size_t(g) + 1] += gptr[size_t(g)];
    {
        std::vector<int32_t> cur(gptr.begin(), gptr.end() - 1);
        for (int64_t i = 0; i < np_; ++i) {
            const int g = int(std::lower_bound(anchors.begin(), anchors.end(), in.anchor[size_t(i)]) - anchors.begin());
            gidx[size_t(cur[size_t(g)]++)] = int32_t(i);
        }
    }
    anchor1_ = ngroups_ == 1 ? anchors[0] : -1;
    if (!counter_.p) {
        counter_.alloc(1);
        TPA_CUDA(cudaMemsetAsync(counter_.p, 0, sizeof(unsigned), s));
    }
    gptr_.upload(gptr.data(), gptr.size(), s);
    gidx_.upload(gidx.data(), gidx.size(), s);
    ganchor_.upload(anchors.data(), anchors.size(), s);
    cptr_.upload(f.coupling.ptr.data(), f.coupling.ptr.size(), s);
    ccol_.upload(f.coupling.col.data(), f.coupling.col.size(), s);
    cval_.upload(f.coupling.val.data(), f.coupling.val.size(), s);
    if (nx_ > 0) {
        // each factor's rows in solve order, entries contiguous per position: the
        // level schedule, or -- when its levels average fewer than 16 rows --
        // plain row order for one thread
        auto lay_out = [&](const CsrRows& m, const LevelSchedule& sc, bool upper, DevBuf<int32_t>& dptr,
                           DevBuf<int32_t>& dcol, DevBuf<double>& dval, DevBuf<int32_t>& dlev,
                           DevBuf<int32_t>& drows, DevBuf<double>* dinv, TriView& view, size_t& bytes) {
            const int levels = sc.levels();
            const bool seq = double(nx_) < 16.0 * double(std::max(levels, 1));
            std::vector<int32_t> order, lev;
            if (seq) {
                for (int64_t i = 0; i < nx_; ++i) order.push_back(int32_t(upper ? nx_ - 1 - i : i));
                lev = {0, int32_t(nx_)};
            } else {
                order = sc.rows;
                lev = sc.level_ptr;
            }
            std::vector<int32_t> ptr(1, 0), col;
            std::vector<double> val, inv;
            for (int32_t k : order) {
                for (int64_t e = m.ptr[size_t(k)]; e < m.ptr[size_t(k) + 1]; ++e) {
                    col.push_back(m.col[size_t(e)]);
                    val.push_back(m.val[size_t(e)]);
                }
                ptr.push_back(int32_t(col.size()));
                if (upper) inv.push_back(1.0 / f.pivot[size_t(k)]);
            }
            dptr.upload(ptr.data(), ptr.size(), s);
            dcol.upload(col.data(), col.size(), s);
            dval.upload(val.data(), val.size(), s);
            dlev.upload(lev.data(), lev.size(), s);
            drows.upload(order.data(), order.size(), s);
            if (dinv) dinv->upload(inv.data(), inv.size(), s);
            view.nlev = int(lev.size()) - 1;
            view.nnz = int(col.size());
            view.seq = seq ? 1 : 0;
            view.lev = dlev.p;
            view.rows = drows.p;
            view.ptr = dptr.p;
            view.col = dcol.p;
            view.val = dval.p;
            view.inv = dinv ? dinv->p : nullptr;
            bytes = col.size() * 8 + (upper ? size_t(nx_) * 8 : 0) +
                    (lev.size() + size_t(nx_) + size_t(nx_) + 1 + col.size()) * 4 + 8;
            llevels_ = upper ? llevels_ : levels;
            ulevels_ = upper ? levels : ulevels_;
        };
        size_t lb = 0, ub = 0;
        lay_out(f.lower, f.lsched, false, lptr_, lcol_, lval_, lsched_, lrows_, nullptr, lview_, lb);
        lay_out(f.upper, f.usched, true, uptr_, ucol_, uval_, usched_, urows_, &piv_, uview_, ub);
        const size_t full = size_t(nx_) * 8 + lb + ub;
        jstaged_ = full <= size_t(200) * 1024 ? 1 : 0;
        jsmem_ = jstaged_ ? full : size_t(nx_) * 8;
        TPA_CUDA(cudaFuncSetAttribute(k_cm_jump_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      int(std::max<size_t>(jsmem_, 1))));
        // the inverses, when the host formed them and two vectors fit in shared memory
        // (TPAGMG_CMDGFM_WALK keeps the row walk, to compare the two paths)
        inverse_ = !f.linv.ptr.empty() && 2 * size_t(nx_) * sizeof(double) <= size_t(200) * 1024 &&
                   !std::getenv("TPAGMG_CMDGFM_WALK");
        if (inverse_) {
            liptr_.upload(f.linv.ptr.data(), f.linv.ptr.size(), s);
            licol_.upload(f.linv.col.data(), f.linv.col.size(), s);
            lival_.upload(f.linv.val.data(), f.linv.val.size(), s);
            uiptr_.upload(f.uinv.ptr.data(), f.uinv.ptr.size(), s);
            uicol_.upload(f.uinv.col.data(), f.uinv.col.size(), s);
            uival_.upload(f.uinv.val.data(), f.uinv.val.size(), s);
            linnz_ = int(f.linv.col.size());
            uinnz_ = int(f.uinv.col.size());
            const size_t vectors = 2 * size_t(nx_) * sizeof(double);
            const size_t entries = (size_t(linnz_) + size_t(uinnz_)) * (sizeof(double) + sizeof(int32_t));
            istaged_ = vectors + entries <= size_t(200) * 1024 ? 1 : 0;
            ismem_ = vectors + (istaged_ ? entries : 0);
            for (ishift_ = 3; ishift_ > 0 && (nx_ << ishift_) > kIluThreads;) --ishift_;
            TPA_CUDA(cudaFuncSetAttribute(k_cm_jump_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          int(ismem_)));
        }
    }
    for (auto* b : {&sol_, &corr_, &x_, &r_, &c_, &p_, &v_, &s_, &t_, &y_, &z_}) b->alloc(size_t(std::max<int64_t>(n_, 1)));
    // cells that are no unknown and no anchor stay zero: the scatter writes the
    // same cells in every iteration
    full_.alloc(size_t(std::max<int64_t>(ncells_, 1)));
    TPA_CUDA(cudaMemsetAsync(full_.p, 0, sizeof(double) * size_t(std::max<int64_t>(ncells_, 1)), s));
    zfull_.alloc(size_t(std::max<int64_t>(ncells_, 1)));
    zp_.alloc(size_t(std::max<int64_t>(np_, 1)));
    partial_.alloc(4 * size_t(kG));
    state_.alloc(kStateSize);
    TPA_CUDA(cudaMemsetAsync(sol_.p, 0, sizeof(double) * size_t(n_), s));
    TPA_CUDA(cudaMemcpyAsync(corr_.p, rhs_.p, sizeof(double) * size_t(n_), cudaMemcpyDeviceToDevice, s));

    const int g = grid_of(n_), ga = grid_of(na_);
    double* p1 = partial_.p;
    double* p2 = partial_.p + kG;
    double* p3 = partial_.p + 2 * kG;
    double* p4 = partial_.p + 3 * kG;
    double hs[kStateSize];
    auto read = [&] {
        TPA_CUDA(cudaMemcpyAsync(hs, state_.p, sizeof(hs), cudaMemcpyDeviceToHost, s));
        TPA_CUDA(cudaStreamSynchronize(s));
    };
    auto defects = [&] {
        k_cm_defects<<<g, kT, 0, s>>>(n_, np_, corr_.p, weight_.p, rows_.p, p1, p2, p3);
        if (na_ > 0)
            k_cm_anchor_defect<<<ga, kT, 0, s>>>(na_, eptr_.p, ecol_.p, eval_.p, erhs_.p, eweight_.p, sol_.p, p4);
        k_cm_defects_fold<<<1, kT, 0, s>>>(p1, p2, p3, g, p4, na_ > 0 ? ga : 0, state_.p);
        launches_ += na_ > 0 ? 3 : 2;
        read();
    };
    auto count = [&](auto launch) {  // a fold of per-block counts
        launch();
        k_cm_sum_fold<<<1, kT, 0, s>>>(p1, g, state_.p + kNorm2);
        launches_ += 2;
        read();
        return hs[kNorm2];
    };
    double rr = 0;
    for (double v : in.rhs) rr += v * v;
    st.initial_residual = std::sqrt(rr);
    const double tol = in.tolerance;
    int iterations = 0;
    if (n_ > 0 && st.initial_residual > 0 && in.warm_start) {
        // `_cmdgfm_initial_solution!` (cmdgfm_projection.jl:1973-2040): zero
        // pressure, then the given previous increment, each with its jumps
        // from the jump factor; the best one that lowers the defect below 0.95
        // of the best so far and the scaled residual norm replaces x = 0
        auto row_defects = [&](const double* res) {
            k_cm_defects<<<g, kT, 0, s>>>(n_, np_, res, weight_.p, rows_.p, p1, p2, p3);
            k_cm_defects_fold<<<1, kT, 0, s>>>(p1, p2, p3, g, p4, 0, state_.p);
            launches_ += 2;
            read();
            const double pd = hs[kPressureDefect], jd = hs[kJumpDefect];
            return std::make_pair((pd != pd || jd != jd) ? NAN : std::max(pd, jd), std::sqrt(hs[kRhsNorm2]));
        };
        if (!ones_.p || ones_.n < size_t(n_)) {
            ones_.alloc(size_t(n_));
            const std::vector<double> one(size_t(n_), 1.0);
            TPA_CUDA(cudaMemcpyAsync(ones_.p, one.data(), sizeof(double) * size_t(n_), cudaMemcpyHostToDevice, s));
            TPA_CUDA(cudaStreamSynchronize(s));
        }
        auto best = row_defects(corr_.p);
        for (int use_previous = 0; use_previous < 2; ++use_previous) {
            TPA_CUDA(cudaMemsetAsync(y_.p, 0, sizeof(double) * size_t(n_), s));
            if (use_previous) {
                if (in.initial.empty()) continue;
                bool any = false, finite = true;
                for (double v : in.initial) {
                    any = any || v != 0.0;
                    finite = finite && std::isfinite(v);
                }
                if (!any || !finite) continue;
                TPA_CUDA(cudaMemcpyAsync(y_.p, in.initial.data(), sizeof(double) * size_t(np_),
                                         cudaMemcpyHostToDevice, s));
            }
            if (nx_ > 0) jump_apply(ds, rhs_.p, ones_.p, ones_.p, y_.p, y_.p, s);
            if (count([&] { k_cm_nonfinite<<<g, kT, 0, s>>>(n_, y_.p, p1); }) != 0.0) continue;
            k_cm_residual<<<g, kT, 0, s>>>(n_, mptr_.p, mcol_.p, mval_.p, rhs_.p, y_.p, t_.p);
            ++launches_;
            const auto cand = row_defects(t_.p);
            if (std::isfinite(cand.first) && std::isfinite(cand.second) && cand.first < 0.95 * best.first &&
                cand.second < best.second) {
                TPA_CUDA(cudaMemcpyAsync(sol_.p, y_.p, sizeof(double) * size_t(n_), cudaMemcpyDeviceToDevice, s));
                best = cand;
                st.initial_guess_used = true;
            }
        }
        k_cm_residual<<<g, kT, 0, s>>>(n_, mptr_.p, mcol_.p, mval_.p, rhs_.p, sol_.p, corr_.p);
        ++launches_;
    }
    if (n_ > 0 && st.initial_residual > 0) {
        while (iterations < in.max_iterations) {
            defects();
            const double pd = hs[kPressureDefect], jd = hs[kJumpDefect], ad = hs[kAnchorDefect];
            const double defect = (pd != pd || jd != jd || ad != ad) ? NAN : std::max(pd, std::max(jd, ad));
            if (!std::isfinite(defect) || defect <= tol) break;
            const double rhs_norm = std::sqrt(hs[kRhsNorm2]);
            if (!std::isfinite(rhs_norm) || rhs_norm == 0.0) break;
            const double requested = std::min(tol, tol / std::max(defect, eps));
            // a tiny correction is normalized before the Krylov run, its scale restored after
            const bool normalize = rhs_norm < 1.0 && rhs_norm * requested < eps;
            const double rhs_scale = normalize ? rhs_norm : 1.0;
            k_cm_scaled_rhs<<<g, kT, 0, s>>>(n_, rows_.p, corr_.p, c_.p, normalize ? 1 : 0, rhs_norm);
            ++launches_;
            int its = bicgstab(ds, in, f, true, requested, in.max_iterations - iterations, s);
            iterations += its;
            ++st.attempts;
            auto nonfinite = [&] {
                return count([&] { k_cm_nonfinite<<<g, kT, 0, s>>>(n_, x_.p, p1); });
            };
            bool finite = nonfinite() == 0.0;
            if (!finite && iterations < in.max_iterations) {
                // the unpreconditioned retry within the remaining budget
                its = bicgstab(ds, in, f, false, requested, in.max_iterations - iterations, s);
                iterations += its;
                ++st.attempts;
                finite = nonfinite() == 0.0;
            }
            if (!finite || its == 0) break;
            const double changed =
                count([&] { k_cm_apply<<<g, kT, 0, s>>>(n_, sol_.p, cols_.p, rhs_scale, x_.p, p1); });
            if (changed == 0.0) break;
            k_cm_residual<<<g, kT, 0, s>>>(n_, mptr_.p, mcol_.p, mval_.p, rhs_.p, sol_.p, corr_.p);
            ++launches_;
        }
    }
    defects();
    st.pressure_defect = hs[kPressureDefect];
    st.jump_defect = hs[kJumpDefect];
    st.anchor_defect = na_ > 0 ? hs[kAnchorDefect] : 0.0;
    st.final_residual = std::sqrt(count([&] { k_cm_norm2<<<g, kT, 0, s>>>(n_, corr_.p, p1); }));
    const double worst = std::max(st.pressure_defect, std::max(st.jump_defect, st.anchor_defect));
    st.converged = std::isfinite(worst) && worst <= tol;
    st.iterations = iterations;
    TPA_CUDA(cudaMemcpyAsync(solution, sol_.p, sizeof(double) * size_t(n_), cudaMemcpyDeviceToHost, s));
    TPA_CUDA(cudaEventRecord(e1, s));
    TPA_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    st.device_ms = ms;
    st.launches = launches_;
    st.inverse = inverse_;
    TPA_CUDA(cudaGetLastError());
}

}  // namespace tpa
