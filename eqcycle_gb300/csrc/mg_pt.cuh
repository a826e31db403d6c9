// Point operations of the vertex levels of the multigrid V-cycle (mg.cu): the 9-point stencil,
// the restriction and prolongation between levels, the first Chebyshev step from x = 0 and the dense
// coarse solve's rows.  Every multiply-add is an explicit round-to-nearest FMA, so any kernel built
// from these functions gives the same bits as the V-cycle's own.  Ld is the load of the vectors the
// V-cycle writes: plain (LdPlain), or the value that a separate kernel would have stored (LdResidual,
// LdProlonged).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "epi.cuh"

namespace eqc {

// Interpolation weights of the GLL nodes k = 0..3 of an element between its lower (lo) and upper (hi)
// vertex along an axis; lo[0] = 1, hi[0] = 0.
template <class T>
struct GllW {
    T lo[4], hi[4];
};

// The restriction from the spectral-element grid by elements: an element's 4 x 4 owned nodes (its local
// indices 0..3; the rest belong to the next element) give each of its four vertices a weighted sum,
// first along a row (lo: towards the lower vertex, hi: the upper one), then over the rows, and a
// vertex adds its elements' four sums.
template <class T>
__device__ __forceinline__ T restrict_lo(const GllW<T>& w, T a0, T a1, T a2, T a3) {
    return fma_rn<T>(w.lo[3], a3, fma_rn<T>(w.lo[2], a2, fma_rn<T>(w.lo[1], a1, a0)));
}
template <class T>
__device__ __forceinline__ T restrict_hi(const GllW<T>& w, T a1, T a2, T a3) {
    return fma_rn<T>(w.hi[3], a3, fma_rn<T>(w.hi[2], a2, mul_rn<T>(w.hi[1], a1)));
}
// the vertex's own element, the one left of it, the one below and the one below left
template <class T>
__device__ __forceinline__ T restrict_sum(T own, T left, T below, T belowleft) {
    return add_rn<T>(add_rn<T>(own, left), add_rn<T>(below, belowleft));
}
// The prolongation's value at local index k of an element with vertex values a (lower) and b (upper).
template <class T>
__device__ __forceinline__ T gll_interp(const GllW<T>& w, int k, T a, T b) {
    return fma_rn<T>(w.hi[k], b, mul_rn<T>(w.lo[k], a));
}

// Ld: the value of a level's vector at grid point (ix, iy).
template <class T>
struct LdPlain {
    const T* p;
    int ld;
    __device__ __forceinline__ T operator()(int ix, int iy) const { return p[(int64_t)iy * ld + ix]; }
};

// The first Chebyshev step from x = 0: x = Dinv b / theta.
template <class T>
__device__ __forceinline__ T cheb_first_pt(T dinv, T b, T inv_theta) { return mul_rn<T>(mul_rn<T>(dinv, b), inv_theta); }

// The coarse level's first step in the restriction that produces its right-hand side.
template <class T>
struct ChebFirst {
    const T* dinv = nullptr;   // null: not fused
    T* x = nullptr;
    T inv_theta = T(0);
};
template <class T>
__device__ __forceinline__ void cheb_first_store(const ChebFirst<T>& F, int64_t i, T b) {
    if (F.dinv) F.x[i] = cheb_first_pt<T>(F.dinv[i], b, F.inv_theta);
}

// Every load below is unconditional (indices clamped into the grid, the weight of a missing neighbour
// zero), so that a point's loads are all in flight together: behind branches they queued up one L2
// latency after another, 8.4 us for a launch whose loads fit in 2.

// (A x) at (ix, iy) of a 9-point stencil level (A[k N + i], offsets (k % 3 - 1, k / 3 - 1)); row 0 is
// the fault row and gives 0, as do neighbours in it.
template <class T>
__device__ __forceinline__ void stencil_row(const T* __restrict__ A, int cx, int cy, int ix, int iy, T (&a)[9]) {
    const int64_t N = (int64_t)cx * cy, i = (int64_t)iy * cx + ix;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int gx = ix + (k % 3) - 1, gy = iy + (k / 3) - 1;
        const T w = __ldg(A + k * N + i);
        a[k] = (gx >= 0 && gx < cx && gy >= 1 && gy < cy) ? w : T(0);
    }
}
template <class T, class V>
__device__ __forceinline__ T stencil_sum(const T (&a)[9], int iy, V v) {
    T s = T(0);
#pragma unroll
    for (int k = 0; k < 9; ++k) s = fma_rn<T>(a[k], v(k), s);
    return iy >= 1 ? s : T(0);
}
template <class T, class Ld>
__device__ __forceinline__ T stencil_pt(const T* __restrict__ A, int cx, int cy, int ix, int iy, Ld x) {
    T a[9], v[9];
    stencil_row<T>(A, cx, cy, ix, iy, a);
#pragma unroll
    for (int k = 0; k < 9; ++k)
        v[k] = x(min(max(ix + (k % 3) - 1, 0), cx - 1), min(max(iy + (k / 3) - 1, 1), cy - 1));
    return stencil_sum<T>(a, iy, [&](int k) { return v[k]; });
}

// Factor-2 coarsening of one axis (make_coarsen_transfer): coarse points at the fine indices 0, 2, 4, ...
// and the last; fine points between two coarse ones take half of each.
struct Coarsen {
    int nf, nc;
    template <class T>
    __device__ __forceinline__ void coarse_of(int i, int& c0, int& c1, T& w0, T& w1) const {
        const bool on = i == nf - 1 || !(i & 1);
        c0 = i == nf - 1 ? nc - 1 : i >> 1;
        c1 = on ? c0 : c0 + 1;
        w0 = on ? T(1) : T(0.5);
        w1 = on ? T(0) : T(0.5);
    }
    // fine point k - 1 left of, on or right of coarse point c (k = 0, 1, 2) and its weight
    template <class T>
    __device__ __forceinline__ int fine_of(int c, int k, T& w) const {
        const int f = min(2 * c, nf - 1), g = f + k - 1;
        w = k == 1 ? T(1) : (k == 0 ? (c > 0 && f == 2 * c ? T(0.5) : T(0)) : (f + 1 < nf - 1 ? T(0.5) : T(0)));
        return min(max(g, 0), nf - 1);
    }
};

// (P xc) at fine point (ix, iy >= 1): the two-by-two bilinear interpolation.
template <class T, class Ld>
__device__ __forceinline__ T prolong_pt(const Coarsen& X, const Coarsen& Y, int ix, int iy, Ld xc) {
    int x0, x1, y0, y1;
    T wx0, wx1, wy0, wy1;
    X.coarse_of<T>(ix, x0, x1, wx0, wx1);
    Y.coarse_of<T>(iy, y0, y1, wy0, wy1);
    const T a = xc(x0, y0), b = xc(x1, y0), c = xc(x0, y1), d = xc(x1, y1);
    const T lo = fma_rn<T>(wx1, b, mul_rn<T>(wx0, a)), hi = fma_rn<T>(wx1, d, mul_rn<T>(wx0, c));
    return fma_rn<T>(wy1, hi, mul_rn<T>(wy0, lo));
}

// The level's residual b - A x, where a separate kernel would have stored it.
template <class T>
struct LdResidual {
    const T *A, *x, *b;
    int cx, cy;
    __device__ __forceinline__ T operator()(int ix, int iy) const {
        return sub_rn<T>(b[(int64_t)iy * cx + ix], stencil_pt<T>(A, cx, cy, ix, iy, LdPlain<T>{x, cx}));
    }
};

// x + P xc, where a separate prolongation would have stored it (rows >= 1).
template <class T>
struct LdProlonged {
    const T *x, *xc;
    Coarsen X, Y;
    __device__ __forceinline__ T operator()(int ix, int iy) const {
        return add_rn<T>(x[(int64_t)iy * X.nf + ix], prolong_pt<T>(X, Y, ix, iy, LdPlain<T>{xc, X.nc}));
    }
};

}  // namespace eqc
