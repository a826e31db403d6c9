// Multigrid V-cycle on the device (see mg.h for the hierarchy).
#include "mg.h"
#include "reduce.cuh"
#include "epi.cuh"
#include "mg_pt.cuh"
#include "sem.h"
#include <algorithm>
#include <cmath>
#include <random>
#include <utility>

namespace eqc {

// ------------------------------------------------------------------ device kernels
// The vertex-level kernels run on 32 x 8 tiles of the grid, one thread per point (no index division).
constexpr int VTX = 32, VTY = 8;

template <class T>
__global__ void __launch_bounds__(VTX * VTY) k_stencil(const T* __restrict__ A, const T* __restrict__ x,
                                                       T* __restrict__ y, int cx, int cy, OpEpi<T> E) {
    EQC_GRID_WAIT();
    const int ix = blockIdx.x * VTX + threadIdx.x, iy = blockIdx.y * VTY + threadIdx.y;
    if (ix >= cx || iy >= cy) return;
    epi_store1(E, y, (int64_t)iy * cx + ix, stencil_pt<T>(A, cx, cy, ix, iy, LdPlain<T>{x, cx}));
}

// Two Chebyshev steps (OpEpi mode 2) in one launch: the first on a tile and the ring around it, one point per
// thread, kept in shared memory, then the second on the tile with the same stencil rows.  A vertex level's
// step is a launch's latency: 3.0 us on 49 x 49 points, and 2.7 for these two.  xp null: the iterate
// before x is 0.  mid (may be null): the first step's iterate.  Points are as k_stencil has them, bit for bit.
// out and mid differ from x and xp, which other tiles' rings read.
template <class T>
__global__ void __launch_bounds__(VTX * VTY) k_stencil2(const T* __restrict__ A, const T* __restrict__ b,
                                                        const T* __restrict__ dinv, const T* __restrict__ x,
                                                        const T* __restrict__ xp, T* __restrict__ mid, T* __restrict__ out,
                                                        int cx, int cy, T c1a, T c2a, T c1b, T c2b) {
    EQC_GRID_WAIT();
    __shared__ T xs[VTY][VTX];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int ix0 = blockIdx.x * (VTX - 2) - 1, iy0 = blockIdx.y * (VTY - 2) - 1;
    const int ix = min(max(ix0 + tx, 0), cx - 1), iy = min(max(iy0 + ty, 0), cy - 1);
    const int64_t i = (int64_t)iy * cx + ix;
    const bool mine = tx > 0 && tx < VTX - 1 && ty > 0 && ty < VTY - 1 && ix0 + tx < cx && iy0 + ty < cy;
    T a[9], v[9];
    stencil_row<T>(A, cx, cy, ix, iy, a);
    const LdPlain<T> ld{x, cx};
#pragma unroll
    for (int k = 0; k < 9; ++k)
        v[k] = ld(min(max(ix + (k % 3) - 1, 0), cx - 1), min(max(iy + (k / 3) - 1, 1), cy - 1));
    const T bi = b[i], di = dinv[i], xi = x[i], xpi = xp ? xp[i] : T(0);
    const T x1 = cheb_x_pt<T>(xi, xpi, bi, stencil_sum<T>(a, iy, [&](int k) { return v[k]; }), di, c1a, c2a);
    xs[ty][tx] = x1;
    __syncthreads();
    if (!mine) return;
    const T t = stencil_sum<T>(a, iy, [&](int k) { return xs[ty + k / 3 - 1][tx + k % 3 - 1]; });
    if (mid) mid[i] = x1;
    out[i] = cheb_x_pt<T>(x1, xi, bi, t, di, c1b, c2b);
}

constexpr int RCX = 15, RCY = 3, RFX = 2 * RCX + 1, RFY = 2 * RCY + 1;
// The sum over a coarse point's 3 x 3 fine points (rs: the tile's residual, RFX x RFY from (2 cx0 - 1, 2 cy0 - 1)).
template <class T>
__device__ __forceinline__ T restrict_tile(const T (&rs)[RFY][RFX], const Coarsen& X, const Coarsen& Y, int cxi, int cyi,
                                           int cx0, int cy0) {
    T s = T(0);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        T w;
        const int gy = Y.fine_of<T>(cyi, q, w);
        T sx = T(0);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            T wx;
            const int gx = X.fine_of<T>(cxi, k, wx);
            sx = fma_rn<T>(wx, rs[min(max(gy - 2 * cy0 + 1, 0), RFY - 1)][min(max(gx - 2 * cx0 + 1, 0), RFX - 1)], sx);
        }
        s = fma_rn<T>(gy == 0 || cyi == 0 ? T(0) : w, sx, s);
    }
    return s;
}

// bc = P^T r on coarse rows >= 1 (row 0 = 0), with the coarse level's first smoothing step, for a tile of
// RCX x RCY coarse points.  One thread per fine point of the tile brings the residual r into shared
// memory: stored by a separate launch (LdPlain), or formed here from the fine operator (LdResidual),
// which saves that launch and r's store and load; the coarse points then sum their 3 x 3 fine points.
template <class T, class Ld>
__global__ void __launch_bounds__(RFX * RFY) k_restrict(Ld rf, T* __restrict__ bc, Coarsen X, Coarsen Y, ChebFirst<T> F) {
    EQC_GRID_WAIT();
    __shared__ T rs[RFY][RFX];
    const int tx = threadIdx.x % RFX, ty = threadIdx.x / RFX;
    const int cx0 = blockIdx.x * RCX, cy0 = blockIdx.y * RCY;
    const int fx = min(max(2 * cx0 - 1 + tx, 0), X.nf - 1), fy = min(max(2 * cy0 - 1 + ty, 0), Y.nf - 1);
    const int cxi = cx0 + threadIdx.x % RCX, cyi = cy0 + threadIdx.x / RCX;
    const bool mine = threadIdx.x < RCX * RCY && cxi < X.nc && cyi < Y.nc;
    const int64_t o = (int64_t)cyi * X.nc + cxi;
    const T di = mine && F.dinv ? F.dinv[o] : T(0);
    rs[ty][tx] = rf(fx, fy);
    __syncthreads();
    if (!mine) return;
    const T s = restrict_tile<T>(rs, X, Y, cxi, cyi, cx0, cy0);
    bc[o] = s;
    if (F.dinv) F.x[o] = cheb_first_pt<T>(di, s, F.inv_theta);
}

// Steps 1 and 2 of the pre-smoothing (k_stencil2 from x1 with the iterate before it 0), the residual of their
// result x3 and its restriction (k_restrict) in one launch: each stage on a ring fewer of the tile's fine
// points, in shared memory.  x3 is stored too, each point by one tile.  3.2 us on 49 x 49 points, where the two
// launches take 2.7 and 2.9: a launch's latency is what a vertex level costs, not the ring's points done twice.
constexpr int RPX = RFX + 4, RPY = RFY + 4;
template <class T>
__global__ void __launch_bounds__(RPX * RPY) k_smooth_restrict(const T* __restrict__ A, const T* __restrict__ b,
                                                               const T* __restrict__ dinv, const T* __restrict__ x1,
                                                               T* __restrict__ x3, T* __restrict__ bc, Coarsen X, Coarsen Y,
                                                               T c1a, T c2a, T c1b, T c2b, ChebFirst<T> F) {
    EQC_GRID_WAIT();
    __shared__ T xs[2][RPY][RPX];
    __shared__ T rs[RFY][RFX];
    const int cx = X.nf, cy = Y.nf;
    const int tx = threadIdx.x % RPX, ty = threadIdx.x / RPX;
    const int cx0 = blockIdx.x * RCX, cy0 = blockIdx.y * RCY;
    const int fx = 2 * cx0 - 3 + tx, fy = 2 * cy0 - 3 + ty;
    const int ix = min(max(fx, 0), cx - 1), iy = min(max(fy, 0), cy - 1);
    const int64_t i = (int64_t)iy * cx + ix;
    const int cxi = cx0 + threadIdx.x % RCX, cyi = cy0 + threadIdx.x / RCX;
    const bool coarse = threadIdx.x < RCX * RCY && cxi < X.nc && cyi < Y.nc;
    const int64_t o = (int64_t)cyi * X.nc + cxi;
    T a[9], v[9];
    stencil_row<T>(A, cx, cy, ix, iy, a);
    const LdPlain<T> ld{x1, cx};
#pragma unroll
    for (int k = 0; k < 9; ++k)
        v[k] = ld(min(max(ix + (k % 3) - 1, 0), cx - 1), min(max(iy + (k / 3) - 1, 1), cy - 1));
    const T bi = b[i], di = dinv[i], xi = x1[i], dc = coarse && F.dinv ? F.dinv[o] : T(0);
    const T x2 = cheb_x_pt<T>(xi, T(0), bi, stencil_sum<T>(a, iy, [&](int k) { return v[k]; }), di, c1a, c2a);
    xs[0][ty][tx] = x2;
    __syncthreads();
    const bool in1 = tx >= 1 && tx < RPX - 1 && ty >= 1 && ty < RPY - 1, in2 = tx >= 2 && tx < RPX - 2 && ty >= 2 && ty < RPY - 2;
    if (in1) {
        const T t = stencil_sum<T>(a, iy, [&](int k) { return xs[0][ty + k / 3 - 1][tx + k % 3 - 1]; });
        const T y = cheb_x_pt<T>(x2, xi, bi, t, di, c1b, c2b);
        xs[1][ty][tx] = y;
        if (fx >= 2 * cx0 && fx < 2 * (cx0 + RCX) && fx < cx && fy >= 2 * cy0 && fy < 2 * (cy0 + RCY) && fy < cy) x3[i] = y;
    }
    __syncthreads();
    if (in2)
        rs[ty - 2][tx - 2] =
            sub_rn<T>(bi, stencil_sum<T>(a, iy, [&](int k) { return xs[1][ty + k / 3 - 1][tx + k % 3 - 1]; }));
    __syncthreads();
    if (!coarse) return;
    const T s = restrict_tile<T>(rs, X, Y, cxi, cyi, cx0, cy0);
    bc[o] = s;
    if (F.dinv) F.x[o] = cheb_first_pt<T>(dc, s, F.inv_theta);
}

// xf = x + P xc on every row (row 0: x)
template <class T>
__global__ void __launch_bounds__(VTX * VTY) k_prolong(T* __restrict__ xf, LdProlonged<T> P) {
    EQC_GRID_WAIT();
    const int ix = blockIdx.x * VTX + threadIdx.x, iy = blockIdx.y * VTY + threadIdx.y;
    if (ix >= P.X.nf || iy >= P.Y.nf) return;
    const int64_t i = (int64_t)iy * P.X.nf + ix;
    xf[i] = iy == 0 ? P.x[i] : P(ix, iy);
}

// The prolongation and the first post-smoothing step in one launch: x' = x + P xc on a tile and the ring
// around it in shared memory, one point per thread, then out = x' + (1 / theta) Dinv (b - A x') on the
// tile; x' is stored too where a second step will need it (xf non-null).
template <class T>
__global__ void __launch_bounds__(VTX * VTY) k_prolong_smooth(const T* __restrict__ A, const T* __restrict__ b,
                                                              const T* __restrict__ dinv, T* __restrict__ xf,
                                                              T* __restrict__ out, LdProlonged<T> P, T inv_theta) {
    EQC_GRID_WAIT();
    __shared__ T xs[VTY][VTX];
    const int cx = P.X.nf, cy = P.Y.nf;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int ix0 = blockIdx.x * (VTX - 2) - 1, iy0 = blockIdx.y * (VTY - 2) - 1;
    const int ix = min(max(ix0 + tx, 0), cx - 1), iy = min(max(iy0 + ty, 0), cy - 1);
    const int64_t i = (int64_t)iy * cx + ix;
    const bool mine = tx > 0 && tx < VTX - 1 && ty > 0 && ty < VTY - 1 && ix0 + tx < cx && iy0 + ty < cy;
    T a[9], bi = T(0), di = T(0);
    if (mine) {
        bi = b[i];
        di = dinv[i];
        stencil_row<T>(A, cx, cy, ix, iy, a);
    }
    const T xi = iy == 0 ? P.x[i] : P(ix, iy);
    xs[ty][tx] = xi;
    __syncthreads();
    if (!mine) return;
    const T t = stencil_sum<T>(a, iy, [&](int k) { return xs[ty + k / 3 - 1][tx + k % 3 - 1]; });
    if (xf) xf[i] = xi;
    out[i] = cheb_x_pt<T>(xi, xi, bi, t, di, T(0), inv_theta);
}

// The prolongation and three post-smoothing steps in one launch (k_prolong_smooth, then k_stencil2 on its result):
// each stage on a ring fewer of the tile's points, in shared memory.  2.9 us on 49 x 49 points, 2.7 and 2.7 apart.
constexpr int PSX = 32, PSY = 16;
template <class T>
__global__ void __launch_bounds__(PSX * PSY) k_prolong_smooth3(const T* __restrict__ A, const T* __restrict__ b,
                                                               const T* __restrict__ dinv, T* __restrict__ out,
                                                               LdProlonged<T> P, T inv_theta, T c1a, T c2a, T c1b, T c2b) {
    EQC_GRID_WAIT();
    __shared__ T xs[2][PSY][PSX];
    const int cx = P.X.nf, cy = P.Y.nf;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int fx = blockIdx.x * (PSX - 6) - 3 + tx, fy = blockIdx.y * (PSY - 6) - 3 + ty;
    const int ix = min(max(fx, 0), cx - 1), iy = min(max(fy, 0), cy - 1);
    const int64_t i = (int64_t)iy * cx + ix;
    T a[9];
    const T bi = b[i], di = dinv[i];
    stencil_row<T>(A, cx, cy, ix, iy, a);
    const int ring = min(min(tx, PSX - 1 - tx), min(ty, PSY - 1 - ty));
    const T x0 = iy == 0 ? P.x[i] : P(ix, iy);
    xs[0][ty][tx] = x0;
    __syncthreads();
    auto at = [&](int s) { return stencil_sum<T>(a, iy, [&](int k) { return xs[s][ty + k / 3 - 1][tx + k % 3 - 1]; }); };
    T y1 = T(0), y2 = T(0);
    if (ring >= 1) xs[1][ty][tx] = y1 = cheb_x_pt<T>(x0, x0, bi, at(0), di, T(0), inv_theta);
    __syncthreads();
    if (ring >= 2) xs[0][ty][tx] = y2 = cheb_x_pt<T>(y1, x0, bi, at(1), di, c1a, c2a);
    __syncthreads();
    if (ring >= 3 && fx < cx && fy < cy) out[i] = cheb_x_pt<T>(y2, y1, bi, at(0), di, c1b, c2b);
}

// ---- transfers between the spectral-element grid and the element-vertex grid ----------
// xf = x + P0 xc; one thread per (vertex column, node row), four nodes each (the last column one).
template <class T>
__global__ void k_prolong_sem(const T* __restrict__ x, const T* __restrict__ xc, T* __restrict__ xf, Layout L, int ldc,
                              GllW<T> w) {
    EQC_GRID_WAIT();
    const int ex = blockIdx.x * blockDim.x + threadIdx.x, iy = blockIdx.y;
    if (ex > L.NelX) return;
    const int ey = iy >> 2, j = iy & 3;
    auto c = [&](int vx, int vy) { return vx <= L.NelX && vy <= L.NelY ? xc[(int64_t)vy * ldc + vx] : T(0); };
    const T a0 = gll_interp(w, j, c(ex, ey), c(ex, ey + 1));
    const T a1 = gll_interp(w, j, c(ex + 1, ey), c(ex + 1, ey + 1));
    const int64_t o = (int64_t)iy * L.ld + 4 * ex;
    xf[o] = add_rn<T>(x[o], a0);
    if (ex == L.NelX) return;
#pragma unroll
    for (int k = 1; k < 4; ++k) xf[o + k] = add_rn<T>(x[o + k], gll_interp(w, k, a0, a1));
}

// bc = P0^T rf over fine rows iy >= 1; coarse row 0 = 0.  One thread per vertex.
template <class T>
__global__ void k_restrict_sem(const T* __restrict__ rf, T* __restrict__ bc, Layout L, int ldc, GllW<T> w,
                               ChebFirst<T> F) {
    EQC_GRID_WAIT();
    const int vx = blockIdx.x * blockDim.x + threadIdx.x;
    const int vy = blockIdx.y;
    if (vx > L.NelX) return;
    // row sums of element (ex, ey): towards its lower (up = 0) or upper vertex
    auto row = [&](int ex, int iy, bool up) {
        T v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int ix = 4 * ex + k;
            v[k] = ix >= 0 && ix < L.nx && iy >= 1 && iy < L.ny ? rf[(int64_t)iy * L.ld + ix] : T(0);
        }
        return up ? restrict_hi(w, v[1], v[2], v[3]) : restrict_lo(w, v[0], v[1], v[2], v[3]);
    };
    T s[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ex = vx - (q & 1), ey = vy - (q >> 1);
        T a[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] = row(ex, 4 * ey + j, q & 1);
        s[q] = (q >> 1) ? restrict_hi(w, a[1], a[2], a[3]) : restrict_lo(w, a[0], a[1], a[2], a[3]);
    }
    const T acc = vy >= 1 ? restrict_sum(s[0], s[1], s[2], s[3]) : T(0);
    bc[(int64_t)vy * ldc + vx] = acc;
    cheb_first_store(F, (int64_t)vy * ldc + vx, acc);
}

// Chebyshev, first step from x = 0: x = Dinv b / theta
template <class T>
__global__ void k_cheb_first(T* __restrict__ x, const T* __restrict__ b, const T* __restrict__ Dinv, int64_t n,
                             T inv_theta) {
    EQC_GRID_WAIT();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = cheb_first_pt<T>(Dinv[i], b[i], inv_theta);
}
// Chebyshev step with t = A x from a separate launch (OpEpi mode 2)
template <class T>
__global__ void k_cheb_step(OpEpi<T> E, const T* __restrict__ t, int64_t n) {
    EQC_GRID_WAIT();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        epi_store1<T>(E, nullptr, i, t[i]);
}
// r = b - t (t may be r)
template <class T>
__global__ void k_sub(const T* __restrict__ b, const T* t, T* r, int64_t n) {
    EQC_GRID_WAIT();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        r[i] = b[i] - t[i];
}
// x[cx + k] = sum_j Cinv[k][j] b[cx + j]  (one warp per row).  Accumulates in T: FP32 for the
// FP32 cycle (a preconditioner; GB300's FP64 rate would make this the slowest kernel of it).
// The right-hand side is staged in shared memory (DNC entries at a time, zero beyond n); each warp reads its row
// in 16-byte loads, asked for before the wait for the kernel that writes b.  FP32: 14 MB at 1,864 unknowns
// from L2, bound by latency, so 16 loads in flight and four rows to a CTA (5.7 us; eight and eight: 7.3).  FP64:
// bound by its arithmetic, eight and eight (13.1 us; sixteen and four with two warps to a row: 15.8).
constexpr int DNC = 2048;
template <class T> constexpr int DN_WARPS = sizeof(T) == 4 ? 4 : 8;
template <class T>
__global__ void __launch_bounds__(32 * DN_WARPS<T>) k_dense_mv(const T* __restrict__ Cinv, const T* __restrict__ b,
                                                               T* __restrict__ x, int n, int pitch, int off) {
    __shared__ __align__(16) T bs[DNC];
    constexpr int V = 16 / (int)sizeof(T), U = sizeof(T) == 4 ? 16 : 8;
    struct alignas(16) Vec { T v[V]; };
    const int lane = threadIdx.x & 31, row = blockIdx.x * DN_WARPS<T> + (threadIdx.x >> 5);
    const T* rw = Cinv + (int64_t)min(row, n - 1) * pitch;
    Vec c[U];
    auto load = [&](int c0) {
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int j = c0 + (q * 32 + lane) * V;
            c[q] = j < pitch ? *reinterpret_cast<const Vec*>(rw + j) : Vec{};
        }
    };
    load(0);
    EQC_GRID_WAIT();
    T s[V];
#pragma unroll
    for (int q = 0; q < V; ++q) s[q] = T(0);
    for (int c0 = 0; c0 < n; c0 += DNC) {
        const int m = min(DNC, pitch - c0);
        if (c0) __syncthreads();
        for (int k = threadIdx.x; k < m; k += 32 * DN_WARPS<T>) bs[k] = c0 + k < n ? b[off + c0 + k] : T(0);
        __syncthreads();
        for (int j0 = 0; j0 < m; j0 += 32 * V * U) {
            if (c0 + j0) load(c0 + j0);
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int j = j0 + (q * 32 + lane) * V;
                if (j >= m) break;
                const Vec d = *reinterpret_cast<const Vec*>(bs + j);
#pragma unroll
                for (int e = 0; e < V; ++e) s[e] = fma_rn<T>(c[q].v[e], d.v[e], s[e]);
            }
        }
    }
    T v = add_rn<T>(s[0], s[1]);
    if constexpr (V == 4) v = add_rn<T>(v, add_rn<T>(s[2], s[3]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = add_rn<T>(v, __shfl_down_sync(0xffffffffu, v, o));
    if (lane == 0 && row < n) x[off + row] = v;
}
template <class T>
__global__ void k_scale(T* x, int64_t n, double s) {
    EQC_GRID_WAIT();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = (T)((double)x[i] * s);
}
template <class T>
__global__ void k_mul(const T* a, T* x, int64_t n) {
    EQC_GRID_WAIT();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = a[i] * x[i];
}

static inline dim3 vgrid2(int cx, int cy) { return dim3((cx + VTX - 1) / VTX, (cy + VTY - 1) / VTY); }
static inline int vb(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 8 * 152); }

// ------------------------------------------------------------------ typed access
template <class T> struct Sel;
template <> struct Sel<double> {
    static double* x(MGWork& w) { return w.x64.p; }
    static double* b(MGWork& w) { return w.b64.p; }
    static double* r(MGWork& w) { return w.r64.p; }
    static double* d(MGWork& w) { return w.d64.p; }
    static double* t(MGWork& w) { return w.t64.p; }
    static const double* A(StencilLevel& l) { return l.A64.p; }
    static const double* Di(StencilLevel& l) { return l.Dinv64.p; }
    static const double* Di0(MGHier& m) { return m.Dinv0_64.p; }
    static const double* C(MGHier& m) { return m.Cinv64.p; }
    static ApplyArgs<double> args(Handle& h) { return args64(h); }
};
template <> struct Sel<float> {
    static float* x(MGWork& w) { return w.x32.p; }
    static float* b(MGWork& w) { return w.b32.p; }
    static float* r(MGWork& w) { return w.r32.p; }
    static float* d(MGWork& w) { return w.d32.p; }
    static float* t(MGWork& w) { return w.t32.p; }
    static const float* A(StencilLevel& l) { return l.A32.p; }
    static const float* Di(StencilLevel& l) { return l.Dinv32.p; }
    static const float* Di0(MGHier& m) { return m.Dinv0_32.p; }
    static const float* C(MGHier& m) { return m.Cinv32.p; }
    static ApplyArgs<float> args(Handle& h) { return args32(h); }
};

template <class T>
static GllW<T> gll_weights(const MGHier& m) {
    GllW<T> g;
    for (int k = 0; k < 4; ++k) {
        g.lo[k] = (T)m.gll_lo[k];
        g.hi[k] = (T)m.gll_hi[k];
    }
    return g;
}

// y = A_l x on level l (0 = spectral-element grid)
template <class T>
static void level_apply(Handle& h, int l, const T* x, T* y) {
    MGHier& m = *h.mg;
    if (l == 0) {
        if constexpr (sizeof(T) == 4) {
            if (sem_usable(h)) {
                SemOp o;
                o.x = x;
                o.out = y;
                sem_launch(h, SL_PLAIN, SE_STORE, SP_NONE, o);
                return;
            }
        }
        apply_K<T>(x, y, Sel<T>::args(h), T(1), 1, h.stream);
    } else {
        StencilLevel& L = m.lev[l - 1];
        k_stencil<T><<<vgrid2(L.cx, L.cy), dim3(VTX, VTY), 0, h.stream>>>(Sel<T>::A(L), x, y, L.cx, L.cy, OpEpi<T>());
        EQC_CHECK_LAUNCH();
        count_launch();
    }
}

// The operator of level l applied to x with the epilogue E (the level's residual or Chebyshev
// step) in the same launch; false when level 0's selected apply kernel has no epilogue.
static bool epi_apply(Handle& h, int l, const float* x, const OpEpi<float>& E) {
    if (!h.fuse) return false;
    if (l == 0) return apply_K_epi(x, args32(h), 1, E, h.stream);
    StencilLevel& L = h.mg->lev[l - 1];
    k_stencil<float><<<vgrid2(L.cx, L.cy), dim3(VTX, VTY), 0, h.stream>>>(L.A32.p, x, nullptr, L.cx, L.cy, E);
    EQC_CHECK_LAUNCH();
    count_launch();
    return true;
}
static bool epi_apply(Handle& h, int l, const double* x, const OpEpi<double>& E) {
    if (!h.fuse) return false;
    if (l == 0) return apply_K_epi(x, args64(h), 1, E, h.stream);
    StencilLevel& L = h.mg->lev[l - 1];
    k_stencil<double><<<vgrid2(L.cx, L.cy), dim3(VTX, VTY), 0, h.stream>>>(L.A64.p, x, nullptr, L.cx, L.cy, E);
    EQC_CHECK_LAUNCH();
    count_launch();
    return true;
}

static int64_t level_size(Handle& h, int l) {
    return l == 0 ? h.L.size() : (int64_t)h.mg->lev[l - 1].cx * h.mg->lev[l - 1].cy;
}

// The Chebyshev smoother's coefficients on level l (0: the spectral-element level): 1/theta of
// the first step and (c1[k], c2[k]) of steps k = 1..deg-1.
static void cheb_coeffs(const MGHier& m, int l, int deg, double* inv_theta, double* c1, double* c2) {
    const double lmax = (l == 0) ? m.lmax0 : m.lev[l - 1].lmax;
    const double lmin = lmax / m.lo_ratio;
    const double theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin);
    const double sigma = theta / delta;
    double rho = 1.0 / sigma;
    *inv_theta = 1.0 / theta;
    for (int k = 1; k < deg; ++k) {
        const double rho_new = 1.0 / (2.0 * sigma - rho);
        c1[k] = rho_new * rho;
        c2[k] = 2.0 * rho_new / delta;
        rho = rho_new;
    }
}

// The level's vectors by their use in one cycle of `deg` smoothing steps each way: the pre-smoothing's
// iterates alternate between post0 and pre and end in pre; the prolongation puts pre + P xc into
// post0, whose post-smoothed iterates alternate between post1 and post0 and end in x (the third
// vector: a launch that forms pre + P xc itself still reads pre around its points).  pairs: the vertex level's
// second and third steps are one launch (k_stencil2), which writes to neither of its operands' vectors.
template <class T>
struct CycleVecs {
    T *pre, *post0, *post1;
    int deg;
    bool pairs;
    T* pre_iter(int k) const { return ((deg - k) & 1) ? post1 : pre; }   // pre-smoothing iterate k = 1..deg
    T* first() const { return pairs ? post1 : pre_iter(1); }
};
template <class T>
static CycleVecs<T> cycle_vecs(const Handle& h, MGWork& w, int l, T* x) {
    const MGHier& m = *h.mg;
    const int deg = std::max(l == 0 ? m.deg : m.deg_coarse, 1);
    const bool even = (deg & 1) == 0;
    return {Sel<T>::t(w), even ? x : Sel<T>::d(w), even ? Sel<T>::d(w) : x, deg, l > 0 && h.fuse && (deg == 3 || deg == 4)};
}

// One Chebyshev step of level l from x (OpEpi mode 2), in the operator's launch where it has the
// epilogue.
template <class T>
static void cheb_step(Handle& h, int l, const T* x, const T* xp, bool xp_zero, T* out, const T* b, T c1, T c2) {
    MGHier& m = *h.mg;
    OpEpi<T> E;
    E.mode = 2;
    E.b = b;
    E.dinv = (l == 0) ? Sel<T>::Di0(m) : Sel<T>::Di(m.lev[l - 1]);
    E.x = x;
    E.xp = xp;
    E.xp_zero = xp_zero;
    E.out = out;
    E.c1 = c1;
    E.c2 = c2;
    if (epi_apply(h, l, x, E)) return;
    T* t = Sel<T>::r(m.work[l]);
    const int64_t n = level_size(h, l);
    level_apply<T>(h, l, x, t);
    k_cheb_step<T><<<vb(n), 256, 0, h.stream>>>(E, t, n);
    EQC_CHECK_LAUNCH();
    count_launch();
}

// Steps 1 and 2 of a vertex level from x (k_stencil2); c1, c2 by step.
template <class T>
static void cheb_pair(Handle& h, int l, const T* x, const T* xp, T* mid, T* out, const T* b, const double* c1,
                      const double* c2) {
    StencilLevel& L = h.mg->lev[l - 1];
    k_stencil2<T><<<dim3((L.cx + VTX - 3) / (VTX - 2), (L.cy + VTY - 3) / (VTY - 2)), dim3(VTX, VTY), 0, h.stream>>>(
        Sel<T>::A(L), b, Sel<T>::Di(L), x, xp, mid, out, L.cx, L.cy, (T)c1[1], (T)c2[1], (T)c1[2], (T)c2[2]);
    EQC_CHECK_LAUNCH();
    count_launch();
}

// The V-cycle on the spectral-element level with its vector work in the operator's launches (sem.cu):
// the first pre-smoothing step and the prolongation are formed as the operand is loaded, the
// residual goes straight into the restriction, and the last launch leaves z.r for the CG.
static void vcycle_sem(Handle& h, float* x, const float* b, CGState* S);

// One V-cycle of level l on A_l x = b from x = 0.  first_done: the restriction that produced b already
// stored the first smoothing step's iterate.
template <class T>
static void vcycle(Handle& h, int l, T* x, const T* b, bool first_done = false) {
    MGHier& m = *h.mg;
    const int L = (int)m.lev.size();
    cudaStream_t s = h.stream;
    if (l == L) {  // coarsest: dense solve on rows >= 1 (row 0 of its vectors stays 0)
        StencilLevel& c = m.lev[L - 1];
        k_dense_mv<T><<<(m.nc + DN_WARPS<T> - 1) / DN_WARPS<T>, 32 * DN_WARPS<T>, 0, s>>>(Sel<T>::C(m), b, x, m.nc, m.nc_pitch, c.cx);
        EQC_CHECK_LAUNCH();
        count_launch();
        return;
    }
    MGWork& w = m.work[l];
    const int64_t n = level_size(h, l);
    const CycleVecs<T> V = cycle_vecs<T>(h, w, l, x);
    std::vector<double> cc1(V.deg), cc2(V.deg);
    double it = 0.0;
    cheb_coeffs(m, l, V.deg, &it, cc1.data(), cc2.data());
    const T inv_theta = (T)it;
    // pre-smoothing from x = 0
    if (!first_done) {
        k_cheb_first<T><<<vb(n), 256, 0, s>>>(V.first(), b, (l == 0) ? Sel<T>::Di0(m) : Sel<T>::Di(m.lev[l - 1]), n,
                                              inv_theta);
        EQC_CHECK_LAUNCH();
        count_launch();
    }
    const bool four = V.deg == 4;
    // three steps with the transfer in one launch; in FP64, whose operations on the rings cost more than a launch on
    // large levels (ms per step of the plain method with them and without: 120 x 240 elements, levels up to
    // 29,161 points, 5.05 and 5.08; 240 x 480, up to 116,161, 13.24 and 13.10; 480 x 960 31.4 and 31.0)
    const bool three = V.pairs && V.deg == 3 && (sizeof(T) == 4 || n <= 40000);
    if (V.pairs && !three) {
        cheb_pair<T>(h, l, V.post1, nullptr, four ? V.pre : nullptr, four ? V.post0 : V.pre, b, cc1.data(), cc2.data());
        if (four) cheb_step<T>(h, l, V.post0, V.pre, false, V.pre, b, (T)cc1[3], (T)cc2[3]);
    } else if (!three) {
        for (int k = 1; k < V.deg; ++k)
            cheb_step<T>(h, l, V.pre_iter(k), k > 1 ? V.pre_iter(k - 1) : nullptr, k == 1, V.pre_iter(k + 1), b, (T)cc1[k],
                         (T)cc2[k]);
    }
    // restriction of the residual b - A x, with the coarse level's first smoothing step (not into the
    // dense level)
    const StencilLevel& lc = m.lev[l];
    MGWork& wc = m.work[l + 1];
    T* bc = Sel<T>::b(wc);
    T* xc = Sel<T>::x(wc);
    ChebFirst<T> F;
    if (l + 1 < L) {
        double itc = 0.0;
        cheb_coeffs(m, l + 1, 1, &itc, nullptr, nullptr);
        F.dinv = Sel<T>::Di(m.lev[l]);
        F.x = cycle_vecs<T>(h, wc, l + 1, xc).first();
        F.inv_theta = (T)itc;
    }
    const dim3 cgrid((lc.cx + RCX - 1) / RCX, (lc.cy + RCY - 1) / RCY);
    const Coarsen X = {l > 0 ? m.lev[l - 1].cx : 0, lc.cx}, Y = {l > 0 ? m.lev[l - 1].cy : 0, lc.cy};   // vertex levels
    if (three) {
        StencilLevel& lev = m.lev[l - 1];
        k_smooth_restrict<T><<<cgrid, RPX * RPY, 0, s>>>(Sel<T>::A(lev), b, Sel<T>::Di(lev), V.post1, V.pre, bc, X, Y, (T)cc1[1],
                                                         (T)cc2[1], (T)cc1[2], (T)cc2[2], F);
    } else if (l > 0 && h.fuse) {
        StencilLevel& lev = m.lev[l - 1];
        k_restrict<T><<<cgrid, RFX * RFY, 0, s>>>(LdResidual<T>{Sel<T>::A(lev), V.pre, b, lev.cx, lev.cy}, bc, X, Y, F);
    } else {
        T* r = Sel<T>::r(w);
        OpEpi<T> E;
        E.mode = 1;
        E.b = b;
        E.out = r;
        if (!epi_apply(h, l, V.pre, E)) {
            level_apply<T>(h, l, V.pre, r);
            k_sub<T><<<vb(n), 256, 0, s>>>(b, r, r, n);
            count_launch();
        }
        if (l == 0)
            k_restrict_sem<T><<<dim3((lc.cx + 127) / 128, lc.cy), 128, 0, s>>>(r, bc, h.L, lc.cx, gll_weights<T>(m), F);
        else
            k_restrict<T><<<cgrid, RFX * RFY, 0, s>>>(LdPlain<T>{r, X.nf}, bc, X, Y, F);
    }
    count_launch();
    EQC_CHECK_LAUNCH();
    vcycle<T>(h, l + 1, xc, bc, l + 1 < L);
    // prolongation and post-smoothing
    if (three) {
        StencilLevel& lev = m.lev[l - 1];
        k_prolong_smooth3<T><<<dim3((lev.cx + PSX - 7) / (PSX - 6), (lev.cy + PSY - 7) / (PSY - 6)), dim3(PSX, PSY), 0, s>>>(
            Sel<T>::A(lev), b, Sel<T>::Di(lev), x, LdProlonged<T>{V.pre, xc, X, Y}, inv_theta, (T)cc1[1], (T)cc2[1], (T)cc1[2],
            (T)cc2[2]);
        EQC_CHECK_LAUNCH();
        count_launch();
        return;
    }
    if (l > 0 && h.fuse) {
        StencilLevel& lev = m.lev[l - 1];
        k_prolong_smooth<T><<<dim3((lev.cx + VTX - 3) / (VTX - 2), (lev.cy + VTY - 3) / (VTY - 2)), dim3(VTX, VTY), 0, s>>>(
            Sel<T>::A(lev), b, Sel<T>::Di(lev), V.deg > 1 ? V.post0 : nullptr, V.pairs ? Sel<T>::r(w) : V.post1,
            LdProlonged<T>{V.pre, xc, X, Y},
            inv_theta);
        count_launch();
    } else {
        if (l == 0)
            k_prolong_sem<T><<<dim3((h.L.NelX + 127) / 128, h.L.ny), 128, 0, s>>>(V.pre, xc, V.post0, h.L, lc.cx,
                                                                                gll_weights<T>(m));
        else
            k_prolong<T><<<vgrid2(X.nf, Y.nf), dim3(VTX, VTY), 0, s>>>(V.post0, LdProlonged<T>{V.pre, xc, X, Y});
        count_launch();
        cheb_step<T>(h, l, V.post0, nullptr, false, V.post1, b, T(0), inv_theta);
    }
    EQC_CHECK_LAUNCH();
    if (V.pairs) {   // the first iterate is in r; the last goes to x, which is post0 for four steps and post1 for three
        cheb_pair<T>(h, l, Sel<T>::r(w), V.post0, four ? V.post1 : nullptr, four ? V.pre : V.post1, b, cc1.data(), cc2.data());
        if (four) cheb_step<T>(h, l, V.pre, V.post1, false, V.post0, b, (T)cc1[3], (T)cc2[3]);
        return;
    }
    for (int k = 1; k < V.deg; ++k) {   // iterate k in post1 (k odd) or post0, the one before it in the other
        T* cur = (k & 1) ? V.post1 : V.post0;
        T* other = (k & 1) ? V.post0 : V.post1;
        cheb_step<T>(h, l, cur, other, false, other, b, (T)cc1[k], (T)cc2[k]);
    }
}

static void vcycle_sem(Handle& h, float* x, const float* b, CGState* S) {
    MGHier& m = *h.mg;
    const int L = (int)m.lev.size();
    MGWork& w = m.work[0];
    MGWork& wc = m.work[1];
    const CycleVecs<float> V = cycle_vecs<float>(h, w, 0, x);
    std::vector<double> cc1(V.deg), cc2(V.deg);
    double it = 0.0;
    cheb_coeffs(m, 0, V.deg, &it, cc1.data(), cc2.data());
    SemOp o;
    o.b = b;
    o.dinv = m.Dinv0_32.p;
    o.inv_theta = (float)it;
    o.w = gll_weights<float>(m);
    if (V.deg == 1) {
        const int64_t n = h.L.size();
        k_cheb_first<float><<<vb(n), 256, 0, h.stream>>>(V.pre, b, o.dinv, n, o.inv_theta);
        EQC_CHECK_LAUNCH();
        count_launch();
    }
    for (int k = 1; k < V.deg; ++k) {
        o.x = V.pre_iter(k);
        o.out = V.pre_iter(k + 1);
        o.xp = k > 2 ? V.pre_iter(k - 1) : nullptr;
        o.c1 = (float)cc1[k];
        o.c2 = (float)cc2[k];
        sem_launch(h, k == 1 ? SL_FIRST : SL_PLAIN, SE_CHEB, k == 1 ? SP_ZERO : (k == 2 ? SP_FIRST : SP_VEC), o);
    }
    o.x = V.pre;
    o.bc = wc.b32.p;
    if (L > 1) {
        double itc = 0.0;
        cheb_coeffs(m, 1, 1, &itc, nullptr, nullptr);
        o.first.dinv = m.lev[0].Dinv32.p;
        o.first.x = cycle_vecs<float>(h, wc, 1, wc.x32.p).first();
        o.first.inv_theta = (float)itc;
    }
    sem_launch(h, SL_PLAIN, SE_RESTRICT, SP_NONE, o);
    vcycle<float>(h, 1, wc.x32.p, wc.b32.p, L > 1);
    o.xc = wc.x32.p;
    o.uout = V.post0;
    o.out = V.post1;
    o.c1 = 0.f;
    o.c2 = (float)it;
    o.S = S;
    o.part = h.red_part.p;
    o.count = h.red_count.p;
    o.dot = V.deg == 1 ? 1 : 0;
    sem_launch(h, SL_PROLONG, SE_CHEB, SP_NONE, o);
    for (int k = 1; k < V.deg; ++k) {   // iterate k in post1 (k odd) or post0, the one before it in the other
        float* other = (k & 1) ? V.post0 : V.post1;
        o.x = (k & 1) ? V.post1 : V.post0;
        o.xp = other;
        o.out = other;
        o.c1 = (float)cc1[k];
        o.c2 = (float)cc2[k];
        o.dot = k + 1 == V.deg ? 1 : 0;
        sem_launch(h, SL_PLAIN, SE_CHEB, SP_VEC, o);
    }
}

// z = M^{-1} r for the CG: r, z are the interior slices (rows >= 1) of level-0 vectors.
void mg_apply64(Handle& h, const double* r, double* z) {
    if (!h.mg) throw Error(EQC_E_STATE, "multigrid not built");
    const int64_t ld = h.L.ld;
    vcycle<double>(h, 0, z - ld, r - ld);
}
bool mg_apply32(Handle& h, const float* r, float* z, CGState* S) {
    if (!h.mg) throw Error(EQC_E_STATE, "multigrid not built");
    const int64_t ld = h.L.ld;
    if (h.fuse && sem_usable(h)) {
        vcycle_sem(h, z - ld, r - ld, S);
        return true;
    }
    vcycle<float>(h, 0, z - ld, r - ld);
    return false;
}

// ------------------------------------------------------------------ setup
static void alloc_work(MGWork& w, int64_t n) {
    for (DBuf<double>* b : {&w.x64, &w.b64, &w.r64, &w.d64, &w.t64}) b->alloc(n);
    for (DBuf<float>* b : {&w.x32, &w.b32, &w.r32, &w.d32, &w.t32}) b->alloc(n);
}

// Largest eigenvalue of D^-1 A_l by power iteration (FP64, 30 steps), times 1.1.
static double estimate_lmax(Handle& h, int l) {
    MGHier& m = *h.mg;
    MGWork& w = m.work[l];
    const int64_t n = level_size(h, l);
    const double* Dinv = (l == 0) ? m.Dinv0_64.p : m.lev[l - 1].Dinv64.p;
    std::vector<double> x0(n);
    std::mt19937_64 rng(1234 + l);
    std::uniform_real_distribution<double> U(0.5, 1.5);
    const int nx = (l == 0) ? h.L.ld : m.lev[l - 1].cx;
    const int nreal = (l == 0) ? h.L.nx : nx;
    for (int64_t i = 0; i < n; ++i) x0[i] = (i < nx || (i % nx) >= nreal) ? 0.0 : U(rng);
    w.x64.upload(x0.data(), n, h.stream);
    double lam = 0.0;
    for (int it = 0; it < 30; ++it) {
        level_apply<double>(h, l, w.x64.p, w.t64.p);
        k_mul<double><<<vb(n), 256, 0, h.stream>>>(Dinv, w.t64.p, n);
        dot64(h, w.t64.p, w.t64.p, n, h.scal.p + 14);
        dot64(h, w.x64.p, w.x64.p, n, h.scal.p + 13);
        double sc[2];
        EQC_CUDA(cudaMemcpyAsync(sc, h.scal.p + 13, sizeof(double) * 2, cudaMemcpyDeviceToHost, h.stream));
        EQC_CUDA(cudaStreamSynchronize(h.stream));
        lam = std::sqrt(sc[1] / sc[0]);
        EQC_CUDA(cudaMemcpyAsync(w.x64.p, w.t64.p, sizeof(double) * n, cudaMemcpyDeviceToDevice, h.stream));
        k_scale<double><<<vb(n), 256, 0, h.stream>>>(w.x64.p, n, 1.0 / std::sqrt(sc[1]));
        count_launch(2);
    }
    EQC_CHECK_LAUNCH();
    return 1.1 * lam;
}

void mg_build(Handle& h) {
    mg_destroy(h);
    h.mg = new MGHier();
    MGHier& m = *h.mg;
    const Layout& L = h.L;
    cudaStream_t s = h.stream;
    static const double xg[5] = {-1.0, -0.65465367070797714, 0.0, 0.65465367070797714, 1.0};
    // level 0 Jacobi scaling
    {
        std::vector<double> dg(L.size());
        h.diag64.download(dg.data(), dg.size(), s);
        EQC_CUDA(cudaStreamSynchronize(s));
        std::vector<double> di(L.size(), 0.0);
        for (int64_t i = L.ld; i < L.size(); ++i) di[i] = ((i % L.ld) < L.nx) ? 1.0 / dg[i] : 0.0;
        std::vector<float> df(di.begin(), di.end());
        m.Dinv0_64.alloc(L.size());
        m.Dinv0_64.upload(di.data(), di.size(), s);
        m.Dinv0_32.alloc(L.size());
        m.Dinv0_32.upload(df.data(), df.size(), s);
    }
    // level 1: vertex grid
    std::vector<double> Wh((size_t)25 * h.Nel);
    h.W64.download(Wh.data(), Wh.size(), s);
    EQC_CUDA(cudaStreamSynchronize(s));
    std::vector<Transfer1D> tx, ty;
    tx.push_back(make_gll_transfer(L.NelX, xg));
    ty.push_back(make_gll_transfer(L.NelY, xg));
    for (int k = 0; k < 4; ++k) {   // weights of local node k (identical in every element)
        m.gll_lo[k] = tx[0].p_w[2 * k];
        m.gll_hi[k] = tx[0].p_w[2 * k + 1];
    }
    StencilLevel l1;
    l1.cx = L.NelX + 1;
    l1.cy = L.NelY + 1;
    l1.A = vertex_operator(h, Wh.data());
    m.lev.push_back(std::move(l1));
    // coarser vertex grids
    const int64_t coarse_max = h.opt.mg_coarse_max > 0 ? h.opt.mg_coarse_max : 2048;
    if (h.opt.mg_degree > 0) m.deg = h.opt.mg_degree;
    m.deg_coarse = h.opt.mg_degree_coarse > 0 ? h.opt.mg_degree_coarse : 3;
    while ((int64_t)m.lev.back().cx * (m.lev.back().cy - 1) > coarse_max && m.lev.back().cx >= 5 &&
           m.lev.back().cy >= 5) {
        StencilLevel& f = m.lev.back();
        Transfer1D ax = make_coarsen_transfer(f.cx), ay = make_coarsen_transfer(f.cy);
        StencilLevel c;
        c.cx = ax.nc;
        c.cy = ay.nc;
        c.A = galerkin_stencil(f.A, f.cx, f.cy, ax, ay, c.cx, c.cy);
        tx.push_back(std::move(ax));
        ty.push_back(std::move(ay));
        m.lev.push_back(std::move(c));
    }
    // upload stencils and diagonal scalings
    for (StencilLevel& lv : m.lev) {
        const size_t N = (size_t)lv.cx * lv.cy;
        std::vector<float> a32(lv.A.begin(), lv.A.end());
        lv.A64.alloc(9 * N);
        lv.A64.upload(lv.A.data(), 9 * N, s);
        lv.A32.alloc(9 * N);
        lv.A32.upload(a32.data(), 9 * N, s);
        std::vector<double> di(N, 0.0);
        for (size_t i = lv.cx; i < N; ++i) di[i] = 1.0 / lv.A[4 * N + i];
        std::vector<float> df(di.begin(), di.end());
        lv.Dinv64.alloc(N);
        lv.Dinv64.upload(di.data(), N, s);
        lv.Dinv32.alloc(N);
        lv.Dinv32.upload(df.data(), N, s);
        EQC_CUDA(cudaStreamSynchronize(s));
    }
    // coarsest dense inverse
    {
        StencilLevel& c = m.lev.back();
        std::vector<double> inv = dense_inverse_spd(c.A, c.cx, c.cy, m.nc);
        m.nc_pitch = (m.nc + 3) / 4 * 4;
        std::vector<double> d((size_t)m.nc * m.nc_pitch, 0.0);
        for (int r = 0; r < m.nc; ++r) std::copy_n(inv.begin() + (size_t)r * m.nc, m.nc, d.begin() + (size_t)r * m.nc_pitch);
        std::vector<float> f(d.begin(), d.end());
        m.Cinv64.alloc(d.size());
        m.Cinv64.upload(d.data(), d.size(), s);
        m.Cinv32.alloc(f.size());
        m.Cinv32.upload(f.data(), f.size(), s);
        EQC_CUDA(cudaStreamSynchronize(s));
    }
    // work vectors
    m.work.resize(m.lev.size() + 1);
    alloc_work(m.work[0], L.size());
    for (size_t k = 0; k < m.lev.size(); ++k) alloc_work(m.work[k + 1], (int64_t)m.lev[k].cx * m.lev[k].cy);
    EQC_CUDA(cudaStreamSynchronize(s));
    // spectral bounds for Chebyshev (all levels but the coarsest, which is solved directly)
    m.lmax0 = estimate_lmax(h, 0);
    for (size_t k = 0; k + 1 < m.lev.size(); ++k) m.lev[k].lmax = estimate_lmax(h, (int)k + 1);
    EQC_CUDA(cudaStreamSynchronize(s));
    // the V-cycle recursion below the coarsest smoothed level uses lev[L-1] as the dense level
}

void mg_clear_work(Handle& h) {
    for (MGWork& w : h.mg->work) {
        for (DBuf<double>* b : {&w.x64, &w.b64, &w.r64, &w.d64, &w.t64}) b->zero(h.stream);
        for (DBuf<float>* b : {&w.x32, &w.b32, &w.r32, &w.d32, &w.t32}) b->zero(h.stream);
    }
}

void mg_destroy(Handle& h) {
    delete h.mg;
    h.mg = nullptr;
}

}  // namespace eqc
