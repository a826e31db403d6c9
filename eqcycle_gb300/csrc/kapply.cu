// K1: matrix-free spectral-element stiffness apply  y = sign * K x.
//
// Replaces the assembled SpMV Ksparse*x of src/main.jl:246,267,311 with the element
// form of src/PCG.jl:82 (element_computation!):
//     a_e = c1 * H * (W_e .* (H' u_e)) + c2 * (W_e .* (u_e H)) * H'
// scattered through the connectivity (the Conn product of src/PCG.jl:266).
//
// GB300 design.  The mesh is structured, so node indices are computed, not loaded; every
// node sums its element contributions in a fixed order (deterministic, no atomics, bitwise
// reproducible).  Per element the work is 5 x-lines and 5 y-lines (sum factorisation: two
// 5-point contractions per line).  Kernels, by apply_variant:
//   k_apply_rows   FP32, one lane per element, one warp per element row, ROWS rows per CTA
//                  plus a halo warp (variants 0, 4-7; the FP32 default);
//   k_apply_walk   the same arithmetic fed by TMA, one wave of CTAs each walking up a strip
//                  (variant 8);
//   k_apply_uni64  FP64: persistent tiles with a TMA pipeline, node-line form, one contraction per
//                  line where the elements have one rigidity (the FP64 default for models of mostly
//                  such elements, classify_elements);
//   k_apply_pipe   the same pipeline with both contractions of every line (variant 3, the FP64 default for
//                  the other models, and the K d refresh of the mixed method's dynamic steps);
//                  k_apply_tma / k_apply_lines: one tile per CTA (1, 2);
//   k_strip        the strip modes 2 and 3 (first element row only).
// Quasi-static solves with variant 0 take their FP32 operator from sem.cu instead.
// The FP32 element kernels take an epilogue (epi.cuh) that finishes the V-cycle's residual or
// Chebyshev step at each owned node.
#include "model.h"
#include "vec.cuh"
#include "epi.cuh"
#include "cg.cuh"
#include <cstdlib>
#include <cmath>
#include <type_traits>
#include <algorithm>

namespace eqc {

__constant__ double cH64[25];  // H[i + 5*j] = h'_i(x_j)
__constant__ float cH32[25];

template <class T> __device__ __forceinline__ T Hc(int i, int j);
template <> __device__ __forceinline__ double Hc<double>(int i, int j) { return cH64[i + 5 * j]; }
template <> __device__ __forceinline__ float Hc<float>(int i, int j) { return cH32[i + 5 * j]; }


// mode 0: full apply, every owned node written
// mode 1: full apply, fault row (iy = 0) written as zero (interior operator K_II)
// mode 2: fault strip: only element row 0, x rows > 0 read as zero, rows 1..4 written
//         (y_I = K_IF x_F, the right-hand side of the quasi-static solve)
// mode 3: fault strip: only element row 0, row 0 written (fault traction (K d)[iFlt])
//
// The strip modes: a thread forms one node column's share of one element (STX elements and the one left of
// them, five columns each), then the columns' nodes sum their one or two elements.  Latency bounds it: every
// thread's loads are independent and its two contractions one chain of FMAs, the x-line of row 0 formed
// again by each of its nodes (mode 3).  240 element columns: 8.0 us as lines through shared
// memory, now 4.2 (mode 2) and 5.6 (mode 3), with the same bits.
constexpr int STX = 8, ST_THREADS = 64;
template <class T, int MODE>
__global__ void __launch_bounds__(ST_THREADS) k_strip(const T* __restrict__ x, T* __restrict__ y, ApplyArgs<T> A, T sign) {
    EQC_GRID_WAIT();
    if (A.gate && *A.gate != A.gate_val) return;
    constexpr int ROWS = MODE == 2 ? 4 : 1, ROW0 = MODE == 2 ? 1 : 0;
    __shared__ T part[ROWS][5 * (STX + 1)];
    const Layout L = A.L;
    const int ex0 = blockIdx.x * STX, t = threadIdx.x, ex = ex0 - 1 + t / 5, i = t % 5;
    if (t < 5 * (STX + 1) && ex >= 0 && ex < L.NelX) {
        const T* w = A.W + (int64_t)ex * 25;
        const T* u = x + 4 * ex;
        T v[5], wy[5], c[5], wx[5];
#pragma unroll
        for (int l = 0; l < 5; ++l) {
            v[l] = MODE == 3 || l == 0 ? u[(int64_t)l * L.ld + i] : T(0);
            wy[l] = w[i + 5 * l];
            if (MODE == 3) {
                c[l] = u[l];
                wx[l] = w[l];
            }
        }
        T s[5];
#pragma unroll
        for (int p = 0; p < 5; ++p) {   // y-line of column i
            T acc = T(0);
#pragma unroll
            for (int l = 0; l < (MODE == 3 ? 5 : 1); ++l) acc = fma_rn<T>(v[l], Hc<T>(l, p), acc);
            s[p] = mul_rn<T>(wy[p], acc);
        }
        T xl = T(0);
        if (MODE == 3) {                // x-line of row 0, at column i
#pragma unroll
            for (int p = 0; p < 5; ++p) {
                T acc = T(0);
#pragma unroll
                for (int k = 0; k < 5; ++k) acc = fma_rn<T>(Hc<T>(k, p), c[k], acc);
                xl = fma_rn<T>(Hc<T>(i, p), mul_rn<T>(wx[p], acc), xl);
            }
            xl = mul_rn<T>((T)A.c1, xl);
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            T acc = T(0);
#pragma unroll
            for (int p = 0; p < 5; ++p) acc = fma_rn<T>(s[p], Hc<T>(ROW0 + r, p), acc);
            part[r][t] = fma_rn<T>((T)A.c2, acc, xl);
        }
    }
    __syncthreads();
    const int nown = ex0 + STX >= L.NelX ? L.nx - 4 * ex0 : 4 * STX;
    for (int k = t; k < nown * ROWS; k += ST_THREADS) {
        const int q = k % nown, r = k / nown, ix = 4 * ex0 + q, e = q / 4 + 1;   // its element, and the one left of it
        T acc = T(0);
        if ((q & 3) == 0) {
            if (ix > 0) acc = add_rn<T>(acc, part[r][5 * (e - 1) + 4]);
            if (ix < L.nx - 1) acc = add_rn<T>(acc, part[r][5 * e]);
        } else {
            acc = add_rn<T>(acc, part[r][5 * e + (q & 3)]);
        }
        y[(int64_t)(ROW0 + r) * L.ld + ix] = sign * acc;
    }
}

// ---------------------------------------------------------------------------------------
// Full apply (modes 0 and 1), node-line formulation.
//
// For a node row iy the x-derivative part of K x is, element column by element column,
//   y1 = c1 * H * (Wrow .* (H' u_row))   with Wrow[p] = sum over the element rows holding iy
// of W_e[p, j_e] (one row inside an element, two on an element boundary: the operator is
// linear in W, so the two element rows collapse into one line).  Likewise every node column
// gives one y-line with the summed W column.  A CTA owns nodes [4ex0, 4ex0+4TEX) x
// [4ey0, 4ey0+4TEY) and runs one x-line item per (owned node row, element column incl. the
// left halo element) and one y-line item per (owned node column, element row incl. the
// bottom halo element).  An item writes its 4 owned outputs and hands the 5th (the shared
// endpoint, owned by the neighbour item) through a small shared array; the final pass adds
// those carries in a fixed order (deterministic, no atomics).  Elements outside the mesh
// act as W = 0, so the one extra CTA row/column that owns the last node line needs no
// special case.
// Even-odd form of the 5-point line contractions (the GLL derivative matrix is centro-
// antisymmetric, D(4-p, 4-k) = -D(p, k)): with e_m = v_m + v_(4-m), o_m = v_m - v_(4-m),
//   s_p, s_(4-p) = P +- Q,  P = sum_m a_pm o_m,  Q = sum_m b_pm e_m + g_p v_2   (p = 0, 1)
//   s_2 = sum_m d_m o_m,    a = (D(p,m) - D(p,4-m)) / 2, b = (D(p,m) + D(p,4-m)) / 2, g = D(p,2),
// 20 operations instead of 25 multiply-adds (Solomonoff's even-odd decomposition of spectral
// differentiation).  EO[0] holds the coefficients of s_p = sum_k H(k,p) v_k (the first
// contraction of a line), EO[1] those of o_i = sum_p H(i,p) s_p (the second).
struct EOCoef {
    float a[2][2], b[2][2], g[2], d[2];
};
struct EOCoef64 {   // the same coefficients for the FP64 kernels
    double a[2][2], b[2][2], g[2], d[2];
};
__constant__ EOCoef cEO[2];
__constant__ EOCoef64 cEO64[2];
__constant__ int cEO_ok;   // H is centro-antisymmetric (else the full contractions are used)

// An element of one rigidity mu has W(p, j) = mu w_p w_j (w the GLL weights), so the two contractions
// of a line and the multiplication between them are one 5 x 5 matrix: the line's share of K x is
// c mu w_j S v with S = D^T diag(w) D.  S is symmetric and centrosymmetric: with o_m = v_m - v_(4-m) and
// e_m = v_m + v_(4-m) - 2 v_2 + g_m v_2,
//   s_p, s_(4-p) = Q +- P,  Q = sum_m b_pm e_m,  P = sum_m a_pm o_m  (p = 0, 1),  s_2 = sum_m d_m e_m,
// 22 operations where the two even-odd contractions and W take 45.  Every entry is taken as a
// difference first (e_m = o_m + 2 (v_(4-m) - v_2)): on a smooth field the differences are exact or
// nearly so, and the rounding left is of the size of the field's variation over the element.
// g (set_H) gives constants the row sums of S, 1e-15 of its entries, that the rounding of the caller's D leaves:
// without it constants would give zero, but the operator would not be the one that the caller's H defines (distance
// from H's operator in extended precision, of the largest |K x|, smooth x on 61 x 95 elements: 6e-15 with both
// contractions, 1e-14 without g; random x 3e-16 any way).
struct UniCoef {
    double a[2][2], b[2][2], d[2], g[2];
    double w[5];
};
__constant__ UniCoef cUni;

__device__ __forceinline__ void uni_line(const double (&v)[5], double (&s)[5]) {
    const double o0 = v[0] - v[4], o1 = v[1] - v[3];
    const double e0 = fma(cUni.g[0], v[2], fma(2.0, v[4] - v[2], o0));
    const double e1 = fma(cUni.g[1], v[2], fma(2.0, v[3] - v[2], o1));
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const double P = fma(cUni.a[p][1], o1, cUni.a[p][0] * o0);
        const double Q = fma(cUni.b[p][1], e1, cUni.b[p][0] * e0);
        s[p] = Q + P;
        s[4 - p] = Q - P;
    }
    s[2] = fma(cUni.d[1], e1, cUni.d[0] * e0);
}

__device__ __forceinline__ void eo5(const float (&v)[5], float (&s)[5], const EOCoef& c) {
    const float e0 = v[0] + v[4], e1 = v[1] + v[3], o0 = v[0] - v[4], o1 = v[1] - v[3];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const float P = fmaf(c.a[p][1], o1, c.a[p][0] * o0);
        const float Q = fmaf(c.g[p], v[2], fmaf(c.b[p][1], e1, c.b[p][0] * e0));
        s[p] = P + Q;
        s[4 - p] = P - Q;
    }
    s[2] = fmaf(c.d[1], o1, c.d[0] * o0);
}

__device__ __forceinline__ void eo5(const double (&v)[5], double (&s)[5], const EOCoef64& c) {
    const double e0 = v[0] + v[4], e1 = v[1] + v[3], o0 = v[0] - v[4], o1 = v[1] - v[3];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const double P = fma(c.a[p][1], o1, c.a[p][0] * o0);
        const double Q = fma(c.g[p], v[2], fma(c.b[p][1], e1, c.b[p][0] * e0));
        s[p] = P + Q;
        s[4 - p] = P - Q;
    }
    s[2] = fma(c.d[1], o1, c.d[0] * o0);
}

// The FP64 node-line kernels take the even-odd contractions where H allows (FP64 issue rate
// bounds them on GB300: 20 operations per contraction instead of 25); the FP32 ones keep the
// full form.
template <class T> __device__ __forceinline__ bool eo_lines() { return false; }
template <> __device__ __forceinline__ bool eo_lines<double>() { return cEO_ok != 0; }
template <class T> struct EOSel;
template <> struct EOSel<float> {
    static __device__ __forceinline__ const EOCoef& c(int k) { return cEO[k]; }
};
template <> struct EOSel<double> {
    static __device__ __forceinline__ const EOCoef64& c(int k) { return cEO64[k]; }
};

// Line items and output pass shared by both full-apply kernels.  us: node tile with row
// pitch UP; ws: element tile, element stride WP, EX elements per row.
template <class T, int TEX, int TEY, int NT, int UP, int WP>
__device__ __forceinline__ void lines_compute(const T* __restrict__ us, const T* __restrict__ ws, T* ys, T* cx,
                                              T* cy, T* __restrict__ y, const ApplyArgs<T>& A, int ex0, int ey0,
                                              T sign, int zero_row0) {
    const Layout& L = A.L;
    constexpr int OX = 4 * TEX, OY = 4 * TEY;
    constexpr int EX = TEX + 1, EY = TEY + 1;
    // x-lines: item = (owned node row r, element column c = 0..TEX, c = 0 the left halo)
    for (int t = threadIdx.x; t < OY * EX; t += NT) {
        const int r = t / EX, c = t - r * EX;
        const int er = (r >> 2) + 1, j = r & 3;
        const T* ul = us + (r + 4) * UP + 4 * c;
        const T* w1 = ws + (er * EX + c) * WP + 5 * j;
        const T* w0 = ws + ((er - 1) * EX + c) * WP + 20;
        T u[5], s[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) u[k] = ul[k];
        T o[5];
        if (eo_lines<T>()) {
            eo5(u, s, EOSel<T>::c(0));
#pragma unroll
            for (int p = 0; p < 5; ++p) s[p] *= (j == 0) ? w1[p] + w0[p] : w1[p];
            eo5(s, o, EOSel<T>::c(1));
#pragma unroll
            for (int i = 0; i < 5; ++i) o[i] = A.c1 * o[i];
        } else {
#pragma unroll
            for (int p = 0; p < 5; ++p) {
                T acc = T(0);
#pragma unroll
                for (int k = 0; k < 5; ++k) acc += Hc<T>(k, p) * u[k];
                const T wr = (j == 0) ? w1[p] + w0[p] : w1[p];
                s[p] = wr * acc;
            }
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                T acc = T(0);
#pragma unroll
                for (int p = 0; p < 5; ++p) acc += Hc<T>(i, p) * s[p];
                o[i] = A.c1 * acc;
            }
        }
        if (c > 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) ys[r * OX + 4 * (c - 1) + i] = o[i];
        }
        cx[r * EX + c] = o[4];
    }
    __syncthreads();
    // y-lines: item = (owned node column q, element row er = 0..TEY, er = 0 the bottom halo)
    for (int t = threadIdx.x; t < EY * OX; t += NT) {
        const int er = t / OX, q = t - er * OX;
        const int ec = (q >> 2) + 1, i = q & 3;
        const T* ul = us + (4 * er) * UP + q + 4;
        const T* w1 = ws + (er * EX + ec) * WP + i;
        const T* w0 = ws + (er * EX + ec - 1) * WP + 4;
        T u[5], s[5];
#pragma unroll
        for (int l = 0; l < 5; ++l) u[l] = ul[l * UP];
        T o[5];
        if (eo_lines<T>()) {
            eo5(u, s, EOSel<T>::c(0));
#pragma unroll
            for (int p = 0; p < 5; ++p) s[p] *= (i == 0) ? w1[5 * p] + w0[5 * p] : w1[5 * p];
            eo5(s, o, EOSel<T>::c(1));
#pragma unroll
            for (int jj = 0; jj < 5; ++jj) o[jj] = A.c2 * o[jj];
        } else {
#pragma unroll
            for (int p = 0; p < 5; ++p) {
                T acc = T(0);
#pragma unroll
                for (int l = 0; l < 5; ++l) acc += u[l] * Hc<T>(l, p);
                const T wc = (i == 0) ? w1[5 * p] + w0[5 * p] : w1[5 * p];
                s[p] = wc * acc;
            }
#pragma unroll
            for (int jj = 0; jj < 5; ++jj) {
                T acc = T(0);
#pragma unroll
                for (int p = 0; p < 5; ++p) acc += s[p] * Hc<T>(jj, p);
                o[jj] = A.c2 * acc;
            }
        }
        if (er > 0) {
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) ys[(4 * (er - 1) + jj) * OX + q] += o[jj];
        }
        cy[er * OX + q] = o[4];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < OY * OX; k += NT) {
        const int r = k / OX, q = k - r * OX;
        const int ix = 4 * ex0 + q, iy = 4 * ey0 + r;
        if (ix >= L.nx || iy >= L.ny) continue;
        T v = ys[k];
        if ((q & 3) == 0) v += cx[r * EX + (q >> 2)];
        if ((r & 3) == 0) v += cy[(r >> 2) * OX + q];
        v = sign * v;
        if (zero_row0 && iy == 0) v = T(0);
        y[(int64_t)iy * L.ld + ix] = v;
    }
}

template <class T, int TEX, int TEY, int NT>
__global__ void __launch_bounds__(NT) k_apply_lines(const T* __restrict__ x, T* __restrict__ y, ApplyArgs<T> A,
                                                    T sign, int zero_row0) {
    EQC_GRID_WAIT();
    if (A.gate && *A.gate != A.gate_val) return;
    const Layout L = A.L;
    constexpr int UX = 4 * TEX + 5, UY = 4 * TEY + 5;   // node tile incl. one halo element
    constexpr int OX = 4 * TEX, OY = 4 * TEY;           // owned nodes
    constexpr int EX = TEX + 1, EY = TEY + 1;           // elements incl. halo
    __shared__ T us[UY * UX];
    __shared__ T ws[EY * EX * 25];
    __shared__ T ys[OY * OX];
    __shared__ T cx[OY * EX];   // x-line endpoint carries [row][element column]
    __shared__ T cy[EY * OX];   // y-line endpoint carries [element row][column]
    const int ex0 = blockIdx.x * TEX, ey0 = blockIdx.y * TEY;
    const int ix0 = 4 * ex0 - 4, iy0 = 4 * ey0 - 4;

    // Issue every tile load of this thread before the first shared-memory store, so that
    // all of them are in flight together (compile-time trip counts, predicated).
    constexpr int NU = (UY * UX + NT - 1) / NT, NWL = (EY * EX * 25 + NT - 1) / NT;
    T ur[NU], wr[NWL];
#pragma unroll
    for (int it = 0; it < NU; ++it) {
        const int k = threadIdx.x + it * NT;
        const int b = k / UX, a = k - b * UX;
        const int ix = ix0 + a, iy = iy0 + b;
        ur[it] = (k < UY * UX && ix >= 0 && ix < L.nx && iy >= 0 && iy < L.ny) ? __ldg(x + (int64_t)iy * L.ld + ix)
                                                                                : T(0);
    }
#pragma unroll
    for (int it = 0; it < NWL; ++it) {
        const int k = threadIdx.x + it * NT;
        const int le = k / 25, q = k - le * 25;
        const int er = le / EX, ec = le - er * EX;
        const int ex = ex0 - 1 + ec, ey = ey0 - 1 + er;
        wr[it] = (k < EY * EX * 25 && ex >= 0 && ex < L.NelX && ey >= 0 && ey < L.NelY)
                     ? __ldg(A.W + ((int64_t)ey * L.NelX + ex) * 25 + q)
                     : T(0);
    }
#pragma unroll
    for (int it = 0; it < NU; ++it) {
        const int k = threadIdx.x + it * NT;
        if (k < UY * UX) us[k] = ur[it];
    }
#pragma unroll
    for (int it = 0; it < NWL; ++it) {
        const int k = threadIdx.x + it * NT;
        if (k < EY * EX * 25) ws[k] = wr[it];
    }
    __syncthreads();

    lines_compute<T, TEX, TEY, NT, UX, 25>(us, ws, ys, cx, cy, y, A, ex0, ey0, sign, zero_row0);
}

// ---- TMA version -------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// 2-D tiled bulk tensor load global -> shared, completion counted on the mbarrier.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

constexpr int UPT = 40;                    // node-tile row pitch of the TMA box (16-byte multiple)

// Full apply with the node tile and the element tile fetched by TMA.  The node box starts at
// x = 4*ex0 - 4 (a multiple of 4 elements, hence 16-byte aligned) and the hardware fills
// coordinates outside the grid with zeros; the element box starts at element ex0 - 1 of a
// copy of W padded to WPad values per element.
template <class T, int TEX, int TEY, int NT>
__global__ void __launch_bounds__(NT) k_apply_tma(const __grid_constant__ CUtensorMap umap,
                                                  const __grid_constant__ CUtensorMap wmap, T* __restrict__ y,
                                                  ApplyArgs<T> A, T sign, int zero_row0) {
    EQC_GRID_WAIT();
    if (A.gate && *A.gate != A.gate_val) return;
    constexpr int UY = 4 * TEY + 5;
    constexpr int OX = 4 * TEX, OY = 4 * TEY;
    constexpr int EX = TEX + 1, EY = TEY + 1;
    constexpr int WP = WPad<T>::v;
    __shared__ __align__(128) T us[UY * UPT];
    __shared__ __align__(128) T ws[EY * EX * WP];
    __shared__ T ys[OY * OX];
    __shared__ T cx[OY * EX];
    __shared__ T cy[EY * OX];
    __shared__ __align__(8) uint64_t bar;
    const int ex0 = blockIdx.x * TEX, ey0 = blockIdx.y * TEY;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, (uint32_t)(sizeof(T) * (UY * UPT + EY * EX * WP)));
        tma_load_2d(us, &umap, &bar, 4 * ex0 - 4, 4 * ey0 - 4);
        tma_load_2d(ws, &wmap, &bar, (ex0 - 1) * WP, ey0 - 1);
    }
    bool done = false;
    for (int it = 0; it < A.wait_polls && !done; ++it) done = mbar_try_wait(&bar, 0);
    if (__syncthreads_or(!done)) {
        // give up (every thread of the CTA alike): flag it, wait (bounded) for the copies still
        // targeting this CTA, leave
        if (threadIdx.x == 0) {
            if (A.err) atomicExch(A.err, 1);
            for (int it = 0; it < MBAR_SPIN_LIMIT; ++it)
                if (mbar_try_wait(&bar, 0)) break;
        }
        return;
    }
    lines_compute<T, TEX, TEY, NT, UPT, WP>(us, ws, ys, cx, cy, y, A, ex0, ey0, sign, zero_row0);
}

// ---- persistent, pipelined version ---------------------------------------------------------
// A grid of a few CTAs per SM walks the tile list (tile t = blockIdx.x + k*gridDim.x); each CTA
// keeps PSTAGES tiles in flight: the node and element tiles of tile i+PSTAGES are fetched by
// TMA while tile i is computed, so HBM streams continuously instead of once per CTA lifetime.
constexpr int PSTAGES = 3;

template <class T, int TEX, int TEY>
struct PipeLayout {
    static constexpr int UY = 4 * TEY + 5, OX = 4 * TEX, OY = 4 * TEY, EX = TEX + 1, EY = TEY + 1;
    static constexpr int WP = WPad<T>::v;
    static constexpr int U_BYTES = UY * UPT * (int)sizeof(T);            // node tile
    static constexpr int W_BYTES = EY * EX * WP * (int)sizeof(T);        // element tile
    static constexpr int STAGE = ((U_BYTES + 127) / 128 + (W_BYTES + 127) / 128) * 128;
    static constexpr int WORK = (OY * OX + OY * EX + EY * OX) * (int)sizeof(T);
    static constexpr int BYTES = PSTAGES * STAGE + ((WORK + 127) / 128) * 128 + 8 * PSTAGES;
};

template <class T, int TEX, int TEY, int NT>
__global__ void __launch_bounds__(NT) k_apply_pipe(const __grid_constant__ CUtensorMap umap,
                                                   const __grid_constant__ CUtensorMap wmap, T* __restrict__ y,
                                                   ApplyArgs<T> A, T sign, int zero_row0, int ntx, int ntiles) {
    EQC_GRID_WAIT();
    if (A.gate && *A.gate != A.gate_val) return;
    using PL = PipeLayout<T, TEX, TEY>;
    extern __shared__ __align__(128) unsigned char smem[];
    T* ys = reinterpret_cast<T*>(smem + PSTAGES * PL::STAGE);
    T* cxs = ys + PL::OY * PL::OX;
    T* cys = cxs + PL::OY * PL::EX;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + PSTAGES * PL::STAGE + ((PL::WORK + 127) / 128) * 128);
    auto us_of = [&](int st) { return reinterpret_cast<T*>(smem + st * PL::STAGE); };
    auto ws_of = [&](int st) { return reinterpret_cast<T*>(smem + st * PL::STAGE + ((PL::U_BYTES + 127) / 128) * 128); };
    auto issue = [&](int t, int st) {
        const int ex0 = (t % ntx) * TEX, ey0 = (t / ntx) * TEY;
        mbar_expect_tx(&bar[st], (uint32_t)(PL::U_BYTES + PL::W_BYTES));
        tma_load_2d(us_of(st), &umap, &bar[st], 4 * ex0 - 4, 4 * ey0 - 4);
        tma_load_2d(ws_of(st), &wmap, &bar[st], (ex0 - 1) * PL::WP, ey0 - 1);
    };
    if (threadIdx.x == 0) {
        for (int st = 0; st < PSTAGES; ++st) mbar_init(&bar[st], 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int st = 0; st < PSTAGES; ++st) {
            const int t = blockIdx.x + st * gridDim.x;
            if (t < ntiles) issue(t, st);
        }
    int i = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++i) {
        const int st = i % PSTAGES;
        const uint32_t parity = (uint32_t)((i / PSTAGES) & 1);
        bool done = false;
        const int polls = i == 0 ? A.wait_polls : MBAR_SPIN_LIMIT;
        for (int it = 0; it < polls && !done; ++it) done = mbar_try_wait(&bar[st], parity);
        if (__syncthreads_or(!done)) {
            // give up: flag it, wait (bounded) for every copy still targeting this CTA, leave
            if (threadIdx.x == 0) {
                if (A.err) atomicExch(A.err, 1);
                int j = i;
                for (int tt = t; tt < ntiles && j < i + PSTAGES; tt += gridDim.x, ++j) {
                    const int sj = j % PSTAGES;
                    const uint32_t pj = (uint32_t)((j / PSTAGES) & 1);
                    for (int it = 0; it < MBAR_SPIN_LIMIT; ++it)
                        if (mbar_try_wait(&bar[sj], pj)) break;
                }
            }
            return;
        }
        const int ex0 = (t % ntx) * TEX, ey0 = (t / ntx) * TEY;
        lines_compute<T, TEX, TEY, NT, UPT, PL::WP>(us_of(st), ws_of(st), ys, cxs, cys, y, A, ex0, ey0, sign,
                                                    zero_row0);
        __syncthreads();   // every thread is done with this stage and with ys/cx/cy
        if (threadIdx.x == 0) {
            const int tn = t + PSTAGES * gridDim.x;
            if (tn < ntiles) issue(tn, st);
        }
    }
}

// ---- FP64: persistent, pipelined, one contraction per line ---------------------------------
// Rigidity of every element with one rigidity (k_classify), -1 for the others, on a grid shifted by
// one column (column ex + 1; zero columns and rows outside the mesh).  An element outside the mesh
// has rigidity 0.
// Tolerance 2^-49: W is a rounded product of weights and rigidity (and of damage factors), a few
// units in the last place from the product formed here.
// mu32: the rigidity over `unit` rounded to FP32; *several counts the elements of several.
__global__ void k_classify(const double* __restrict__ W, double* __restrict__ mu, float* __restrict__ mu32, int* several,
                           int NelX, int NelY, int pitch, double unit, int ok) {
    EQC_GRID_WAIT();
    const int64_t Nel = (int64_t)NelX * NelY;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < Nel; e += (int64_t)gridDim.x * blockDim.x) {
        const double* w = W + 25 * e;
        const double m = w[12] / (cUni.w[2] * cUni.w[2]);
        bool uni = ok && m > 0 && isfinite(m);
        for (int j = 0; j < 5; ++j)
            for (int i = 0; i < 5; ++i)
                uni = uni && fabs(w[i + 5 * j] - m * (cUni.w[i] * cUni.w[j])) <= 0x1p-49 * w[i + 5 * j];
        mu[(e / NelX) * pitch + e % NelX + 1] = uni ? m : -1.0;
        mu32[e] = uni ? (float)(m / unit) : -1.f;
        if (!uni) atomicAdd(several, 1);
    }
}

// *count += the tiles of tx x ty owned elements (on the grid of the element vertices, one halo column and row below
// and left) that hold an element of several rigidities.
__global__ void k_classify_tiles(const double* __restrict__ mu, int pitch, int NelX, int NelY, int tx, int ty, int* count) {
    EQC_GRID_WAIT();
    const int ntx = NelX / tx + 1, ntiles = ntx * (NelY / ty + 1);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x) {
        const int ex0 = (t % ntx) * tx, ey0 = (t / ntx) * ty;
        bool several = false;
        for (int ey = max(ey0 - 1, 0); ey < min(ey0 + ty, NelY); ++ey)
            for (int ex = max(ex0 - 1, 0); ex < min(ex0 + tx, NelX); ++ex) several = several || mu[(int64_t)ey * pitch + ex + 1] < 0.0;
        if (several) atomicAdd(count, 1);
    }
}

// Two contractions with W between them: a line that meets an element of several rigidities.
__device__ __forceinline__ void generic_line(const double (&u)[5], const double (&w)[5], double (&o)[5]) {
    double s[5];
    if (cEO_ok) {
        eo5(u, s, cEO64[0]);
#pragma unroll
        for (int p = 0; p < 5; ++p) s[p] *= w[p];
        eo5(s, o, cEO64[1]);
        return;
    }
#pragma unroll
    for (int p = 0; p < 5; ++p) {
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < 5; ++k) acc += Hc<double>(k, p) * u[k];
        s[p] = w[p] * acc;
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        double acc = 0.0;
#pragma unroll
        for (int p = 0; p < 5; ++p) acc += Hc<double>(i, p) * s[p];
        o[i] = acc;
    }
}

// Tile of 7 x 8 elements by 256 threads: 32 owned node rows times 8 element columns (the left halo
// column first) are one x-line a thread, four whole rows to a warp, so that a line's 5th output
// reaches its owner, the next lane, by a shuffle; 9 element rows (the halo row below first) times 28
// owned node columns are one y-line a thread.
constexpr int UEX = 7, UEY = 8, UNT = 256;
struct UniTile {
    static constexpr int UX = 4 * UEX + 8, UY = 4 * UEY + 5;   // node box (33 of 36 columns used)
    static constexpr int OX = 4 * UEX, OY = 4 * UEY, EX = UEX + 1, EY = UEY + 1;
    static constexpr int MX = 10;                             // rigidity box, from an even column
    static constexpr int U_BYTES = UY * UX * 8, M_BYTES = EY * MX * 8;
    static constexpr int M_OFF = (U_BYTES + 127) / 128 * 128;
    static constexpr int STAGE = M_OFF + (M_BYTES + 127) / 128 * 128;
    static constexpr int YS_OFF = PSTAGES * STAGE, CY_OFF = YS_OFF + OY * OX * 8, BAR_OFF = CY_OFF + EY * OX * 8;
    static constexpr int BYTES = BAR_OFF + 8 * PSTAGES;
};
static_assert(UniTile::OY * UniTile::EX == UNT && UniTile::EY * UniTile::OX <= UNT, "one line of each kind per thread");

// y = sign K x in FP64 (zero_row0: K_II), tiles and stages as k_apply_pipe's, in node lines: a line
// whose one or two elements have one rigidity each takes uni_line, scaled by sign c w_j times their
// summed rigidity (w_0 = w_4); any other line reads its W and takes both contractions.
// Bound: GB300 issues two FP64 operations per SM and clock (every FP64 instruction of a warp holds
// the pipe for 16 clocks, whatever its active lanes), so the lines, their scaling and the sums at
// shared nodes are arranged in whole warps, the rigidities' signs are tested as integers, and a tile
// takes about 460 warp instructions of the pipe: 8.2 per element, where both contractions took 15.
// Back to back on the damage-zone models, before (both contractions, 8 x 7 tiles) and now: 61 x 95
// elements 19.2 and 10.8 us, 120 x 240 37.2 and 22.6, 240 x 480 134.3 and 71.5 (122.8 and 62.5 where
// one x and y stay in L2), 480 x 960 496 and 261: 51 us of the 62.5 are the pipe's.
// TAIL: NoTail; ResidualOut, the mixed solver's residual r64 = -K_II x with its work (sign -1, zero_row0);
// DotOut, the CG's x . K x (a launch of its own took 9 us on 120 x 240 elements, the sum here 1).
struct NoTail {};
template <class TAIL>
__global__ void __launch_bounds__(UNT) k_apply_uni64(const __grid_constant__ CUtensorMap umap,
                                                     const __grid_constant__ CUtensorMap mmap, double* __restrict__ y,
                                                     ApplyArgs<double> A, double sign, int zero_row0, int ntx, int ntiles,
                                                     OpEpi<double> E, TAIL R) {
    EQC_GRID_WAIT();
    if (A.gate && *A.gate != A.gate_val) return;
    constexpr bool RES = std::is_same_v<TAIL, ResidualOut>, DOT = std::is_same_v<TAIL, DotOut>;
    double sg = 0.0;
    int es = 0;
    if constexpr (RES) {
        sg = R.S->sigma;
        es = R.S->sigma_exp;
    }
    DotAcc<std::conditional_t<RES, float, double>> acc;
    using UT = UniTile;
    const Layout& L = A.L;
    extern __shared__ __align__(128) unsigned char smem[];
    double* ys = reinterpret_cast<double*>(smem + UT::YS_OFF);
    double* cy = reinterpret_cast<double*>(smem + UT::CY_OFF);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + UT::BAR_OFF);
    auto issue = [&](int t, int st) {
        const int ex0 = (t % ntx) * UEX, ey0 = (t / ntx) * UEY;
        mbar_expect_tx(&bar[st], (uint32_t)(UT::U_BYTES + UT::M_BYTES));
        tma_load_2d(smem + st * UT::STAGE, &umap, &bar[st], 4 * ex0 - 4, 4 * ey0 - 4);
        tma_load_2d(smem + st * UT::STAGE + UT::M_OFF, &mmap, &bar[st], ex0 & ~1, ey0 - 1);   // 16-byte aligned
    };
    if (threadIdx.x == 0) {
        for (int st = 0; st < PSTAGES; ++st) mbar_init(&bar[st], 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int st = 0; st < PSTAGES; ++st) {
            const int t = blockIdx.x + st * gridDim.x;
            if (t < ntiles) issue(t, st);
        }
    // this thread's x-line (node row r, element column c) and y-line (element row er, node column q)
    const int r = threadIdx.x >> 3, c = threadIdx.x & 7, jx = r & 3;
    const int er = threadIdx.x / UT::OX, q = threadIdx.x - er * UT::OX, kq = q & 3, ec = (q >> 2) + 1;
    const bool has_y = er < UT::EY;
    const double kx = sign * A.c1 * cUni.w[jx], ky = sign * A.c2 * cUni.w[kq];
    // W(p, j) of element (ex, ey), zero outside the mesh
    auto Wat = [&](int ex, int ey, int n) {
        const bool in = ex >= 0 && ex < L.NelX && ey >= 0 && ey < L.NelY;
        return in ? __ldg(A.W + ((int64_t)ey * L.NelX + ex) * 25 + n) : 0.0;
    };
    int i = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++i) {
        const int st = i % PSTAGES;
        const uint32_t parity = (uint32_t)((i / PSTAGES) & 1);
        bool done = false;
        const int polls = i == 0 ? A.wait_polls : MBAR_SPIN_LIMIT;
        for (int it = 0; it < polls && !done; ++it) done = mbar_try_wait(&bar[st], parity);
        done = __all_sync(0xffffffffu, done);   // lanes poll apart: the tile may land between their last polls
        const int ex0 = (t % ntx) * UEX, ey0 = (t / ntx) * UEY;
        const double* us = reinterpret_cast<const double*>(smem + st * UT::STAGE);
        const double* ms = reinterpret_cast<const double*>(smem + st * UT::STAGE + UT::M_OFF) + (ex0 & 1);
        if (done) {
            const double* ul = us + (r + 4) * UT::UX + 4 * c;
            const double2 a = reinterpret_cast<const double2*>(ul)[0], b = reinterpret_cast<const double2*>(ul)[1];
            const double u[5] = {a.x, a.y, b.x, b.y, ul[4]};
            double s[5], kap;
            const double* m = ms + ((r >> 2) + 1) * UT::MX + c;
            const double m1 = m[0], m0 = jx == 0 ? m[-UT::MX] : 0.0;
            if ((__double2hiint(m1) | __double2hiint(m0)) >= 0) {
                uni_line(u, s);
                kap = kx * (m1 + m0);
            } else {
                double w[5];
                const int ex = ex0 - 1 + c, ey = ey0 + (r >> 2);
#pragma unroll
                for (int p = 0; p < 5; ++p) {
                    w[p] = Wat(ex, ey, p + 5 * jx);
                    if (jx == 0) w[p] += Wat(ex, ey - 1, p + 20);
                }
                generic_line(u, w, s);
                kap = sign * A.c1;
            }
            const double carry = __shfl_up_sync(0xffffffffu, kap * s[4], 1);   // of column c - 1
            if (c > 0) {
                double2* o = reinterpret_cast<double2*>(ys + r * UT::OX + 4 * (c - 1));
                o[0] = make_double2(fma(kap, s[0], carry), kap * s[1]);
                o[1] = make_double2(kap * s[2], kap * s[3]);
            }
        }
        if (__syncthreads_or(!done)) {
            // give up: flag it, wait (bounded) for every copy still targeting this CTA, leave
            if (threadIdx.x == 0) {
                if (A.err) atomicExch(A.err, 1);
                int j = i;
                for (int tt = t; tt < ntiles && j < i + PSTAGES; tt += gridDim.x, ++j)
                    for (int it = 0; it < MBAR_SPIN_LIMIT; ++it)
                        if (mbar_try_wait(&bar[j % PSTAGES], (uint32_t)((j / PSTAGES) & 1))) break;
            }
            break;
        }
        double v[4];
        if (has_y) {
            const double* ul = us + (4 * er) * UT::UX + q + 4;
            double u[5], s[5], kap;
#pragma unroll
            for (int l = 0; l < 5; ++l) u[l] = ul[l * UT::UX];
            const double* m = ms + er * UT::MX + ec;
            const double m1 = m[0], m0 = kq == 0 ? m[-1] : 0.0;
            if ((__double2hiint(m1) | __double2hiint(m0)) >= 0) {
                uni_line(u, s);
                kap = ky * (m1 + m0);
            } else {
                double w[5];
                const int ex = ex0 - 1 + ec, ey = ey0 - 1 + er;
#pragma unroll
                for (int p = 0; p < 5; ++p) {
                    w[p] = Wat(ex, ey, kq + 5 * p);
                    if (kq == 0) w[p] += Wat(ex - 1, ey, 4 + 5 * p);
                }
                generic_line(u, w, s);
                kap = sign * A.c2;
            }
            cy[er * UT::OX + q] = kap * s[4];
            if (er > 0) {
#pragma unroll
                for (int l = 0; l < 4; ++l) v[l] = fma(kap, s[l], ys[(4 * (er - 1) + l) * UT::OX + q]);
            }
        }
        // the epilogue's operands, in flight across the barrier
        const int ix = 4 * ex0 + q, iy0 = 4 * (ey0 + er - 1);
        const bool mine = has_y && er > 0 && ix < L.nx;
        const int64_t o0 = (int64_t)iy0 * L.ld + ix;
        EpiIn<double> in[4];
        double xin[4];
        if (mine && !RES) {
#pragma unroll
            for (int l = 0; l < 4; ++l)
                if (iy0 + l < L.ny) {
                    if constexpr (DOT) xin[l] = E.x[o0 + (int64_t)l * L.ld];
                    else in[l] = epi_load1(E, o0 + (int64_t)l * L.ld);
                }
        }
        __syncthreads();   // cy written; every read of this stage and of ys done
        if (threadIdx.x == 0) {
            const int tn = t + PSTAGES * gridDim.x;
            if (tn < ntiles) issue(tn, st);
        }
        if (mine) {
            v[0] += cy[(er - 1) * UT::OX + q];
#pragma unroll
            for (int l = 0; l < 4; ++l)
                if (iy0 + l < L.ny) {
                    const int64_t o = o0 + (int64_t)l * L.ld;
                    const double t = (zero_row0 && iy0 + l == 0) ? 0.0 : v[l];
                    if constexpr (DOT) {
                        y[o] = t;
                        acc.add(t, xin[l]);
                    } else if constexpr (RES) {
                        R.r64[o] = t;
                        R.r32[o] = residual32(t, es, sg, acc);
                    } else {
                        epi_finish1(E, y, o, t, in[l]);
                    }
                }
        }
    }
    if constexpr (RES) residual_done(R, acc);
    if constexpr (DOT) grid_sum(acc, R.part, R.count, [&](double t) { cg_take_dot(R.S, t, true); });
}

// ---- element-per-lane version (FP32) --------------------------------------------------------
// One lane per element, one warp per element row of 31 elements plus a halo lane (lane 0 = the
// element left of the strip), ROWS element rows per CTA plus a halo warp (warp 0 = the row
// below the group).  Every lane contracts its element's 5 x-lines and 5 y-lines in registers
// (no W merging across elements): the 4 x 4 nodes it owns (local i, j < 4) are complete once the
// right-column contributions of the left lane (shuffle) and the top-row contributions of the warp
// below (shared memory, one barrier) are added.  Node rows arrive as 16-byte loads (the 5th node
// of a row is the next lane's first), element data as seven 16-byte loads of the padded W copy.
// The last node row and column are owned by a virtual element row / column with W = 0.
constexpr unsigned FULLMASK = 0xffffffffu;

// The 5 x-lines and 5 y-lines of one element (u: its 5 x 5 nodes, W: its 25 weights): the owned
// outputs out[j][i] (i, j < 4), the right column R[j] (j < 4) and the top row T[i] (i <= 4).
// top_only: only T is needed (the halo row).
template <class WAcc>
__device__ __forceinline__ void rows_lines_t(const float (&u)[5][5], const WAcc& W, float c1, float c2,
                                           bool top_only, float (&out)[4][4], float (&R)[4], float (&T)[5]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) out[j][i] = 0.f;
    // x-lines (the halo warp needs only the top one)
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        if (top_only && j < 4) continue;
        float sp[5];
#pragma unroll
        for (int p = 0; p < 5; ++p) {
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < 5; ++k) acc += Hc<float>(k, p) * u[j][k];
            sp[p] = W[p + 5 * j] * acc;
        }
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            float acc = 0.f;
#pragma unroll
            for (int p = 0; p < 5; ++p) acc += Hc<float>(i, p) * sp[p];
            const float o = c1 * acc;
            if (j < 4) {
                if (i < 4) out[j][i] = o;
                else R[j] = o;
            } else {
                T[i] = o;
            }
        }
    }
    // y-lines
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        float sp[5];
#pragma unroll
        for (int p = 0; p < 5; ++p) {
            float acc = 0.f;
#pragma unroll
            for (int l = 0; l < 5; ++l) acc += u[l][i] * Hc<float>(l, p);
            sp[p] = W[i + 5 * p] * acc;
        }
#pragma unroll
        for (int jj = 0; jj < 5; ++jj) {
            float acc = 0.f;
#pragma unroll
            for (int p = 0; p < 5; ++p) acc += sp[p] * Hc<float>(jj, p);
            const float o = c2 * acc;
            if (jj < 4) {
                if (i < 4) out[jj][i] += o;
                else R[jj] += o;
            } else {
                T[i] += o;
            }
        }
    }
}

__device__ __forceinline__ void rows_lines_eo(const float (&u)[5][5], const float (&W)[28], float c1, float c2,
                                              bool top_only, float (&out)[4][4], float (&R)[4], float (&T)[5]) {
    // x-lines
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        if (top_only && j < 4) {   // the halo row needs only its top row T
#pragma unroll
            for (int i = 0; i < 4; ++i) out[j][i] = 0.f;
            R[j] = 0.f;
            continue;
        }
        float s[5], o[5];
        eo5(u[j], s, cEO[0]);
#pragma unroll
        for (int p = 0; p < 5; ++p) s[p] *= W[p + 5 * j];
        eo5(s, o, cEO[1]);
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const float v = c1 * o[i];
            if (j < 4) {
                if (i < 4) out[j][i] = v;
                else R[j] = v;
            } else {
                T[i] = v;
            }
        }
    }
    // y-lines
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        float v[5], s[5], o[5];
#pragma unroll
        for (int l = 0; l < 5; ++l) v[l] = u[l][i];
        eo5(v, s, cEO[0]);
#pragma unroll
        for (int p = 0; p < 5; ++p) s[p] *= W[i + 5 * p];
        eo5(s, o, cEO[1]);
#pragma unroll
        for (int jj = 0; jj < 5; ++jj) {
            if (top_only && jj < 4) continue;
            const float w = c2 * o[jj];
            if (jj < 4) {
                if (i < 4) out[jj][i] += w;
                else R[jj] += w;
            } else {
                T[i] += w;
            }
        }
    }
}

__device__ __forceinline__ void rows_lines(const float (&u)[5][5], const float (&W)[28], float c1, float c2,
                                           bool top_only, float (&out)[4][4], float (&R)[4], float (&T)[5]) {
    if (cEO_ok) rows_lines_eo(u, W, c1, c2, top_only, out, R, T);
    else rows_lines_t(u, W, c1, c2, top_only, out, R, T);
}

template <int ROWS, int MINB>
__global__ void __launch_bounds__(32 * (ROWS + 1), MINB) k_apply_rows(const float* __restrict__ x, float* __restrict__ y,
                                                                     ApplyArgs<float> A, float sign, int zero_row0,
                                                                     OpEpi<float> E) {
    const Layout L = A.L;
    __shared__ float Ts[ROWS + 1][5][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ex = (int)blockIdx.x * 31 - 1 + lane;
    const int ey = (int)blockIdx.y * ROWS - 1 + w;
    const bool real = ex >= 0 && ex < L.NelX && ey >= 0 && ey < L.NelY;
    // the element data are constant (written only between launches, by the host): their loads
    // are issued before the wait for the grids this launch depends on, so they overlap the
    // predecessor's tail when the launch is programmatic
    float4 wq[7];
    const float4* wp = reinterpret_cast<const float4*>(A.Wp + ((int64_t)(real ? ey : 0) * L.NelX + (real ? ex : 0)) * 28);
#pragma unroll
    for (int k = 0; k < 7; ++k) wq[k] = real ? __ldg(wp + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    EQC_GRID_WAIT();
    if (A.gate && *A.gate != A.gate_val) return;

    // every load of the lane is issued before the first use (one memory latency, not twelve)
    float4 v[5];
    float n4s[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const int iy = 4 * ey + j;
        const bool rowok = iy >= 0 && iy < L.ny;
        v[j] = (rowok && ex >= 0 && 4 * ex < L.nx) ? __ldg(reinterpret_cast<const float4*>(x + (int64_t)iy * L.ld + 4 * ex))
                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
        const int ix = 4 * ex + 4;
        n4s[j] = (lane == 31 && rowok && ix >= 0 && ix < L.nx) ? __ldg(x + (int64_t)iy * L.ld + ix) : 0.f;
    }
    float u[5][5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        u[j][0] = v[j].x;
        u[j][1] = v[j].y;
        u[j][2] = v[j].z;
        u[j][3] = v[j].w;
        const float n4 = __shfl_down_sync(FULLMASK, v[j].x, 1);
        u[j][4] = lane == 31 ? n4s[j] : n4;
    }
    float W[28];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        W[4 * k] = wq[k].x;
        W[4 * k + 1] = wq[k].y;
        W[4 * k + 2] = wq[k].z;
        W[4 * k + 3] = wq[k].w;
    }

    float out[4][4], R[4], T[5];
    rows_lines(u, W, A.c1, A.c2, w == 0, out, R, T);
#pragma unroll
    for (int i = 0; i < 5; ++i) Ts[w][i][lane] = T[i];
    float Rl[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) Rl[j] = __shfl_up_sync(FULLMASK, R[j], 1);
    __syncthreads();
    if (w == 0 || lane == 0 || ex > L.NelX || ey > L.NelY) return;
    // contributions of the left element (right column) and of the element row below (top row)
#pragma unroll
    for (int j = 0; j < 4; ++j) out[j][0] += Rl[j];
#pragma unroll
    for (int i = 0; i < 4; ++i) out[0][i] += Ts[w - 1][i][lane];
    out[0][0] += Ts[w - 1][4][lane - 1];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int iy = 4 * ey + j;
        if (iy >= L.ny) break;
        const float z = (zero_row0 && iy == 0) ? 0.f : sign;
        epi_store4(E, y, (int64_t)iy * L.ld + 4 * ex,
                   make_float4(z * out[j][0], z * out[j][1], z * out[j][2], z * out[j][3]),
                   make_float4(u[j][0], u[j][1], u[j][2], u[j][3]));
    }
}

// ---- element-per-lane apply fed by TMA, walking up the strips (FP32) ------------------------
// The grid is one wave (every CTA resident at once).  CTA b walks strip b % nsx (31 element
// columns plus the halo lane) upward through element rows [r0, r0 + rw) in tiles of 8 element
// rows, one per warp (warps past the walk's last row sit the last tile out).  Each tile's node rows (one 132 x 33 box) and element
// records (one 28 x 32 x 8 box of the padded W copy) arrive by TMA into one of two stages while
// the other stage's tile is computed, so a CTA never waits on memory between its tiles.  In the
// first tile warp 0 computes the row below the walk (top row only: the halo); in later tiles the
// row below warp 0 is the previous tile's warp 7, whose top-row contributions are carried in
// shared memory.  Coordinates outside the mesh read as zero (virtual elements have W = 0).  The
// arithmetic and the order of the carries are those of k_apply_rows: both give the same bits.
constexpr int WK_ROWS = 8, WK_UX = 132, WK_UY = 4 * WK_ROWS + 1;
constexpr int WK_U_BYTES = WK_UX * WK_UY * 4;                     // 17,424
constexpr int WK_W_BYTES = 28 * 32 * WK_ROWS * 4;                 // 28,672
constexpr int WK_W_OFF = ((WK_U_BYTES + 127) / 128) * 128;
constexpr int WK_STAGE = WK_W_OFF + WK_W_BYTES;
constexpr int WK_TS_OFF = 2 * WK_STAGE;                           // [2][ROWS][5][32] floats
constexpr int WK_BAR_OFF = WK_TS_OFF + 2 * WK_ROWS * 5 * 32 * 4;
constexpr int WK_BYTES = WK_BAR_OFF + 16;

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
// orders this thread's earlier generic-proxy shared-memory accesses before later TMA writes
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__global__ void __launch_bounds__(32 * WK_ROWS, 2) k_apply_walk(const __grid_constant__ CUtensorMap umap,
                                                                const __grid_constant__ CUtensorMap wmap,
                                                                float* __restrict__ y, ApplyArgs<float> A, float sign,
                                                                int zero_row0, int nsx, int rw, OpEpi<float> E) {
    extern __shared__ __align__(128) unsigned char smem[];
    const Layout L = A.L;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ex0 = 31 * ((int)blockIdx.x % nsx);   // element of lane 1
    const int r0 = ((int)blockIdx.x / nsx) * rw;
    const int r_end = min(r0 + rw, L.NelY + 1);     // element row NelY is the virtual top row
    const int nt = (r_end - r0 + WK_ROWS) / WK_ROWS;  // tiles cover rows r0 - 1 .. r_end - 1
    float* Ts = reinterpret_cast<float*>(smem + WK_TS_OFF);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + WK_BAR_OFF);
    auto issue_w = [&](int k) {   // element records of tile k; the barrier expects the node rows too
        const int st = k & 1, base = r0 - 1 + WK_ROWS * k;
        mbar_expect_tx(&bar[st], (uint32_t)(WK_U_BYTES + WK_W_BYTES));
        tma_load_3d(smem + st * WK_STAGE + WK_W_OFF, &wmap, &bar[st], 0, ex0 - 1, base);
    };
    auto issue_u = [&](int k) {   // node rows of tile k
        const int st = k & 1, base = r0 - 1 + WK_ROWS * k;
        tma_load_2d(smem + st * WK_STAGE, &umap, &bar[st], 4 * (ex0 - 1), 4 * base);
    };
    auto issue = [&](int k) {
        issue_w(k);
        issue_u(k);
    };
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
    }
    __syncthreads();
    // the element data are constant (written only between launches, by the host): the first
    // tile's records are requested before the wait for the grids this launch depends on, so they
    // stream in during the predecessor's tail when the launch is programmatic; the node rows (the
    // predecessor's output) after it.  The first tile alone: it reaches every CTA before any
    // second one.
    // A gated launch (A.gate) requests nothing before the wait: it may have no work.
    const bool gated = A.gate != nullptr;
    if (threadIdx.x == 0 && !gated) issue_w(0);
    EQC_GRID_WAIT();
    if (gated && *A.gate != A.gate_val) return;
    if (threadIdx.x == 0) {
        if (gated) issue_w(0);
        issue_u(0);
    }
    const int ex = ex0 - 1 + lane;
    for (int k = 0; k < nt; ++k) {
        const int st = k & 1;
        const uint32_t parity = (uint32_t)((k >> 1) & 1);
        bool done = false;
        const int polls = k == 0 ? A.wait_polls : MBAR_SPIN_LIMIT;
        for (int it = 0; it < polls && !done; ++it) done = mbar_try_wait(&bar[st], parity);
        if (__syncthreads_or(!done)) {
            // give up: flag it, wait (bounded) for the copies still in flight (tile 0, or tiles
            // k and k + 1), leave
            if (threadIdx.x == 0) {
                if (A.err) atomicExch(A.err, 1);
                for (int j = k; j < nt && j < (k == 0 ? 1 : k + 2); ++j)
                    for (int it = 0; it < MBAR_SPIN_LIMIT; ++it)
                        if (mbar_try_wait(&bar[j & 1], (uint32_t)((j >> 1) & 1))) break;
            }
            return;
        }
        if (k == 0 && nt > 1 && threadIdx.x == 0) issue(1);   // overlaps the first tile's compute
        const int ey = r0 - 1 + WK_ROWS * k + w;
        if (ey >= r_end) {   // past the walk (warp-uniform): no row to compute, only the barrier
            __syncthreads();
            if (threadIdx.x == 0 && k + 2 < nt) {
                fence_proxy_async_smem();
                issue(k + 2);
            }
            continue;
        }
        const float* xs = reinterpret_cast<const float*>(smem + st * WK_STAGE) + 4 * w * WK_UX;
        const float* wsm = reinterpret_cast<const float*>(smem + st * WK_STAGE + WK_W_OFF) + (w * 32 + lane) * 28;
        float u[5][5];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(xs + j * WK_UX + 4 * lane);
            u[j][0] = v.x;
            u[j][1] = v.y;
            u[j][2] = v.z;
            u[j][3] = v.w;
            const float n4 = __shfl_down_sync(FULLMASK, v.x, 1);
            u[j][4] = lane == 31 ? xs[j * WK_UX + 128] : n4;
        }
        float W[28];
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            const float4 c = *reinterpret_cast<const float4*>(wsm + 4 * q);
            W[4 * q] = c.x;
            W[4 * q + 1] = c.y;
            W[4 * q + 2] = c.z;
            W[4 * q + 3] = c.w;
        }
        const bool halo = k == 0 && w == 0;
        float out[4][4], R[4], T[5];
        rows_lines(u, W, A.c1, A.c2, halo, out, R, T);
        float* Tk = Ts + st * (WK_ROWS * 160);
#pragma unroll
        for (int i = 0; i < 5; ++i) Tk[(w * 5 + i) * 32 + lane] = T[i];
        float Rl[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) Rl[j] = __shfl_up_sync(FULLMASK, R[j], 1);
        // warp 0 after the first tile: the top row of the previous tile's warp 7 (written before
        // the previous tile's barrier, overwritten only after this tile's)
        float cb[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
        if (w == 0 && k > 0) {
            const float* Tp = Ts + (st ^ 1) * (WK_ROWS * 160) + (WK_ROWS - 1) * 160;
#pragma unroll
            for (int i = 0; i < 4; ++i) cb[i] = Tp[i * 32 + lane];
            cb[4] = Tp[4 * 32 + (lane > 0 ? lane - 1 : 0)];
        }
        __syncthreads();   // T of every warp written; every read of this stage done
        if (threadIdx.x == 0 && k + 2 < nt) {
            fence_proxy_async_smem();
            issue(k + 2);
        }
        if (lane == 0 || halo || ex > L.NelX || ey > L.NelY || ey >= r_end) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) out[j][0] += Rl[j];
        if (w > 0) {
            const float* Tb = Tk + (w - 1) * 160;
#pragma unroll
            for (int i = 0; i < 4; ++i) out[0][i] += Tb[i * 32 + lane];
            out[0][0] += Tb[4 * 32 + lane - 1];
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) out[0][i] += cb[i];
            out[0][0] += cb[4];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int iy = 4 * ey + j;
            if (iy >= L.ny) break;
            const float z = (zero_row0 && iy == 0) ? 0.f : sign;
            epi_store4(E, y, (int64_t)iy * L.ld + 4 * ex,
                       make_float4(z * out[j][0], z * out[j][1], z * out[j][2], z * out[j][3]),
                       make_float4(u[j][0], u[j][1], u[j][2], u[j][3]));
        }
    }
}

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                     const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static PFN_encodeTiled encode_fn() {
    static PFN_encodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_encodeTiled)p;
    }
    return fn;
}

static bool encode_2d(CUtensorMap* m, bool f64, const void* base, uint64_t d0, uint64_t d1, uint64_t stride_bytes,
                      uint32_t b0, uint32_t b1) {
    PFN_encodeTiled fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {d0, d1};
    const cuuint64_t strides[1] = {stride_bytes};
    const cuuint32_t box[2] = {b0, b1};
    const cuuint32_t es[2] = {1, 1};
    return fn(m, f64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base),
              dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// W of the walk apply as a 3-D tensor [NelY][NelX][28] with a 28 x 32 x WK_ROWS box.
static bool encode_w_walk(CUtensorMap* m, const float* base, int NelX, int NelY) {
    PFN_encodeTiled fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {28, (cuuint64_t)NelX, (cuuint64_t)NelY};
    const cuuint64_t strides[2] = {28 * sizeof(float), (cuuint64_t)NelX * 28 * sizeof(float)};
    const cuuint32_t box[3] = {28, 32, WK_ROWS};
    const cuuint32_t es[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int LTEX = 8, LTEY = 7, LNT = 256;

template <class T> static CUtensorMap& wmap_ref(TmaCache& c);
template <> CUtensorMap& wmap_ref<float>(TmaCache& c) { return c.w32; }
template <> CUtensorMap& wmap_ref<double>(TmaCache& c) { return c.w64; }
template <class T> static std::unordered_map<const void*, CUtensorMap>& umap_ref(TmaCache& c);
template <> std::unordered_map<const void*, CUtensorMap>& umap_ref<float>(TmaCache& c) { return c.u32; }
template <> std::unordered_map<const void*, CUtensorMap>& umap_ref<double>(TmaCache& c) { return c.u64; }

template <class T>
static const CUtensorMap& tma_wmap(TmaCache& c) { return wmap_ref<T>(c); }

// Tensor map of a node vector (cached by address): the nx x ny grid, row pitch ld, box
// UPT x (4*LTEY+5); coordinates outside the grid read as zero.
template <class T>
static const CUtensorMap* tma_umap(TmaCache& c, const T* x, const Layout& L) {
    if (!c.ok) return nullptr;
    auto& m = umap_ref<T>(c);
    auto it = m.find(x);
    if (it != m.end()) return &it->second;
    if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) return nullptr;
    CUtensorMap tm;
    if (!encode_2d(&tm, sizeof(T) == 8, x, (uint64_t)L.nx, (uint64_t)L.ny, (uint64_t)L.ld * sizeof(T), UPT,
                   4 * LTEY + 5))
        return nullptr;
    return &(m[x] = tm);
}

// Node-vector map of k_apply_uni64 (cached by address).
static const CUtensorMap* tma_umap_uni(TmaCache& c, const double* x, const Layout& L) {
    if (!c.ok) return nullptr;
    auto it = c.u64uni.find(x);
    if (it != c.u64uni.end()) return &it->second;
    if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) return nullptr;
    CUtensorMap tm;
    if (!encode_2d(&tm, true, x, (uint64_t)L.nx, (uint64_t)L.ny, (uint64_t)L.ld * sizeof(double), UniTile::UX, UniTile::UY))
        return nullptr;
    return &(c.u64uni[x] = tm);
}

// Node-vector map of the walk apply (cached by address): box WK_UX x WK_UY.
static const CUtensorMap* tma_umap_walk(TmaCache& c, const float* x, const Layout& L) {
    if (!c.walk_ok) return nullptr;
    auto it = c.u32walk.find(x);
    if (it != c.u32walk.end()) return &it->second;
    if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) return nullptr;
    CUtensorMap tm;
    if (!encode_2d(&tm, false, x, (uint64_t)L.nx, (uint64_t)L.ny, (uint64_t)L.ld * sizeof(float), WK_UX, WK_UY))
        return nullptr;
    return &(c.u32walk[x] = tm);
}

// Encodes the element-data maps of the padded W copies W32p / W64p; leaves the cache disabled
// (plain loads) if TMA is unavailable.
void tma_init_for(TmaCache& c, const Layout& L, const float* W32p, const double* W64p, const double* mu) {
    c.ok = false;
    c.walk_ok = false;
    c.u32.clear();
    c.u64.clear();
    c.u32walk.clear();
    c.u64uni.clear();
    if (getenv("EQC_NO_TMA")) return;
    const int EX = LTEX + 1, EY = LTEY + 1;
    bool ok = encode_2d(&c.w32, false, W32p, (uint64_t)L.NelX * WPad<float>::v, (uint64_t)L.NelY,
                        (uint64_t)L.NelX * WPad<float>::v * sizeof(float), EX * WPad<float>::v, EY);
    ok = ok && encode_2d(&c.w64, true, W64p, (uint64_t)L.NelX * WPad<double>::v, (uint64_t)L.NelY,
                         (uint64_t)L.NelX * WPad<double>::v * sizeof(double), EX * WPad<double>::v, EY);
    const int mp = mu_pitch(L.NelX);
    ok = ok && encode_2d(&c.mu, true, mu, (uint64_t)mp, (uint64_t)L.NelY, (uint64_t)mp * sizeof(double), UniTile::MX,
                         UniTile::EY);
    c.ok = ok;
    c.walk_ok = ok && encode_w_walk(&c.w32walk, W32p, L.NelX, L.NelY);
}
void tma_init(Handle& h) { tma_init_for(h.tma, h.L, h.W32p.p, h.W64p.p, h.mu64.p); }

void classify_elements(Handle& h) {
    const Layout& L = h.L;
    const int mp = mu_pitch(L.NelX);
    const int64_t Nel = (int64_t)L.NelX * L.NelY;
    if (!h.mu64.p) h.mu64.alloc((size_t)mp * L.NelY);
    if (!h.mu32.p) h.mu32.alloc(Nel);
    if (h.mu_unit == 0.0) {
        double w = 0.0;
        EQC_CUDA(cudaMemcpyAsync(&w, h.W64.p + 25 * (Nel - 1) + 12, sizeof(w), cudaMemcpyDeviceToHost, h.stream));
        EQC_CUDA(cudaStreamSynchronize(h.stream));
        w /= (32.0 / 45.0) * (32.0 / 45.0);
        h.mu_unit = w > 0.0 && std::isfinite(w) ? w : 1.0;
    }
    DBuf<int> several;   // elements, tiles of the FP64 apply and of the double-float one
    several.alloc(3);
    k_classify<<<(int)std::min<int64_t>((Nel + 255) / 256, 4096), 256, 0, h.stream>>>(
        h.W64.p, h.mu64.p, h.mu32.p, several.p, L.NelX, L.NelY, mp, h.mu_unit, h.uni_ok ? 1 : 0);
    const int64_t t64 = (int64_t)(L.NelX / UEX + 1) * (L.NelY / UEY + 1), tdf = (int64_t)(L.NelX / DF_COLS + 1) * (L.NelY / DF_ROWS + 1);
    k_classify_tiles<<<(int)std::min<int64_t>((t64 + 255) / 256, 4096), 256, 0, h.stream>>>(h.mu64.p, mp, L.NelX, L.NelY, UEX, UEY,
                                                                                         several.p + 1);
    k_classify_tiles<<<(int)std::min<int64_t>((tdf + 255) / 256, 4096), 256, 0, h.stream>>>(h.mu64.p, mp, L.NelX, L.NelY, DF_COLS,
                                                                                         DF_ROWS, several.p + 2);
    EQC_CHECK_LAUNCH();
    count_launch(3);
    int n[3] = {0, 0, 0};
    several.download(n, 3, h.stream);
    EQC_CUDA(cudaStreamSynchronize(h.stream));
    // The one-contraction FP64 apply against the pipeline with both contractions, by the share f of its tiles that hold
    // an element of several rigidities (us a launch, x and y in L2, 240 x 480 elements; before the line 135 for any f):
    // none 70 and 135; scattered, f = 0.5 94 and 135, 0.77 105, 0.9 113, 0.99 134, then up to 170; in a band 87 at
    // f = 0.25, 98 at 0.45, 110 at 0.66.  On 120 x 240: none 22 and 39, f = 0.5 31 and 39, 0.89 36, 0.99 41, up to 50; a
    // band 36 at f = 0.66 and 40 at 0.75.  So up to two thirds of the tiles.  With two tiles or fewer to an SM the
    // slowest tile sets the time: 61 x 95 in bands of 3 % 14 and 15, of 6 % 16 and 15, of 25 % 19 and 15; one
    // element in 32 is asked there too.
    const int64_t several_el = n[0];
    h.uni64_pays = h.uni_ok && 3 * (int64_t)n[1] <= 2 * t64 && (t64 > 2 * 152 || 32 * several_el <= Nel);
    h.few_several = 128 * several_el <= Nel;   // for df_pays
    // The double-float apply (240 x 480): none 37 us, scattered over 0.28 of the CTAs 59, 0.36 62, 0.5 68, and 67 with
    // both contractions everywhere.
    h.uni_df_pays = h.uni_ok && 5 * (int64_t)n[2] <= 2 * tdf;
    // The operator of sem.cu against the row-tile apply with its vector kernels (ms per quasi-static step, elements of
    // several rigidities scattered over the mesh, whose warps take both contractions): one in eight 3.16 on 240 x 480
    // elements and 9.33 on 480 x 960; one in four 3.24 and 3.41, 9.38 and 10.96; all 1.21 and 1.37 on 48 x 48, 1.66
    // and 1.83 on 120 x 240, 3.31 and 3.49, 9.39 and 10.97.  It was the faster one at every share: one in eight keeps
    // models of mostly several rigidities on the apply that the Newmark steps use.
    h.sem_ok = h.uni_ok && several_el * 8 <= Nel && L.size() < (int64_t)1 << 29 &&   // 32-bit byte offsets
               L.NelX < 31 * 4096;                                              // partials of a dot product's CTAs
}

// CTAs of the pipelined apply: as many as fit on every SM at once.
static int g_pipe_blocks[2] = {0, 0};
template <class T>
static int pipe_blocks() { return g_pipe_blocks[sizeof(T) == 8 ? 1 : 0]; }

// CTAs that fit with `bytes` of shared memory each; `most`: the most that a launch asks for.  A kernel's limit is set
// to one value only: another thread may be launching it while this one creates a handle.
template <class K>
static int resident_blocks(K kernel, int threads, int bytes, int most = 0) {
    EQC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(bytes, most)));
    int per_sm = 0, dev = 0, nsm = 0;
    EQC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, bytes));
    EQC_CUDA(cudaGetDevice(&dev));
    EQC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    return std::max(1, per_sm) * nsm;
}

// Launch shape of k_apply_uni64: g_uni_sms SMs, at most g_uni_per_sm CTAs on each.
static int g_uni_sms = 0;
template <class TAIL> static int g_uni_per_sm = 0;
constexpr int UNI_SMEM = 120 * 1024;   // the most a CTA asks for: then one fits an SM
static void uni_setup() {
    int dev = 0;
    EQC_CUDA(cudaGetDevice(&dev));
    EQC_CUDA(cudaDeviceGetAttribute(&g_uni_sms, cudaDevAttrMultiProcessorCount, dev));
    auto one = [](auto kernel, int& per_sm) {
        per_sm = resident_blocks(kernel, UNT, UniTile::BYTES, UNI_SMEM) / g_uni_sms;
    };
    one(k_apply_uni64<NoTail>, g_uni_per_sm<NoTail>);
    one(k_apply_uni64<ResidualOut>, g_uni_per_sm<ResidualOut>);
    one(k_apply_uni64<DotOut>, g_uni_per_sm<DotOut>);
}
// The FP64 pipe of each SM bounds the kernel, so its CTAs have to be spread evenly: per SM no more than
// an even spread of the tiles needs, kept to that by the shared memory that a CTA asks for.  (A
// programmatic launch otherwise fills the SMs that its predecessor leaves empty with several CTAs
// each: 26 us instead of 16 back to back on 61 x 95 elements.)
template <class TAIL = NoTail>
static void launch_uni64(const CUtensorMap& um, double* y, const ApplyArgs<double>& A, double sign, int zr,
                         cudaStream_t s, const OpEpi<double>& E = OpEpi<double>(), const TAIL& R = TAIL()) {
    const int ntx = A.L.NelX / UEX + 1, ntiles = ntx * (A.L.NelY / UEY + 1);
    const int per_sm = std::min(g_uni_per_sm<TAIL>, (ntiles + g_uni_sms - 1) / g_uni_sms);
    const int smem = std::max(UniTile::BYTES, std::min(UNI_SMEM, 228 * 1024 / (per_sm + 1) / 128 * 128 + 128));
    const int grid = std::min(ntiles, per_sm * g_uni_sms);
    k_apply_uni64<TAIL><<<grid, UNT, smem, s>>>(um, A.tma->mu, y, A, sign, zr, ntx, ntiles, E, R);
    EQC_CHECK_LAUNCH();
    count_launch();
}

// CTAs of the walk apply that are resident at once (its grid never exceeds one wave).
static int g_walk_slots = 0;

// Walk length: the rows of every strip split evenly over the resident CTAs (one wave, every
// SM holding the same number of rows to within one walk).
static void walk_shape(const Layout& L, int* nsx, int* rw, int* nblk) {
    *nsx = (L.NelX + 1 + 30) / 31;
    const int64_t rows = L.NelY + 1;
    int64_t r = std::max<int64_t>(1, (rows * *nsx + g_walk_slots - 1) / g_walk_slots);
    while (r < rows && *nsx * ((rows + r - 1) / r) > g_walk_slots) ++r;
    *rw = (int)r;
    *nblk = *nsx * (int)((rows + r - 1) / r);
}

static bool launch_walk(const float* x, float* y, const ApplyArgs<float>& A, float sign, int zr, cudaStream_t s,
                        const OpEpi<float>& E = OpEpi<float>()) {
    if (!A.tma || !A.tma->walk_ok || g_walk_slots <= 0) return false;
    const CUtensorMap* um = tma_umap_walk(*A.tma, x, A.L);
    if (!um) return false;
    int nsx, rw, nblk;
    walk_shape(A.L, &nsx, &rw, &nblk);
    k_apply_walk<<<nblk, 32 * WK_ROWS, WK_BYTES, s>>>(*um, A.tma->w32walk, y, A, sign, zr, nsx, rw, E);
    EQC_CHECK_LAUNCH();
    count_launch();
    return true;
}

bool set_H(const double* H, cudaStream_t s) {
    float hf[25];
    bool uni = false;
    for (int k = 0; k < 25; ++k) hf[k] = (float)H[k];
    EQC_CUDA(cudaMemcpyToSymbolAsync(cH64, H, sizeof(double) * 25, 0, cudaMemcpyHostToDevice, s));
    EQC_CUDA(cudaMemcpyToSymbolAsync(cH32, hf, sizeof(float) * 25, 0, cudaMemcpyHostToDevice, s));
    {   // even-odd coefficients of the two line contractions (H[i + 5 j] = h'_i(x_j))
        auto D1 = [&](int p, int k) { return H[k + 5 * p]; };   // s_p = sum_k H(k,p) v_k
        auto D2 = [&](int i, int p) { return H[i + 5 * p]; };   // o_i = sum_p H(i,p) s_p
        double hmax = 0.0, asym = 0.0;
        for (int k = 0; k < 25; ++k) hmax = std::max(hmax, std::fabs(H[k]));
        for (int i = 0; i < 5; ++i)
            for (int j = 0; j < 5; ++j) asym = std::max(asym, std::fabs(H[i + 5 * j] + H[(4 - i) + 5 * (4 - j)]));
        EOCoef c[2];
        for (int t = 0; t < 2; ++t) {
            auto M = [&](int r, int q) { return t == 0 ? D1(r, q) : D2(r, q); };
            for (int p = 0; p < 2; ++p) {
                for (int m = 0; m < 2; ++m) {
                    c[t].a[p][m] = (float)(0.5 * (M(p, m) - M(p, 4 - m)));
                    c[t].b[p][m] = (float)(0.5 * (M(p, m) + M(p, 4 - m)));
                }
                c[t].g[p] = (float)M(p, 2);
                c[t].d[p] = (float)M(2, p);
            }
        }
        EOCoef64 c64[2];
        for (int t = 0; t < 2; ++t) {
            auto M = [&](int r, int q) { return t == 0 ? D1(r, q) : D2(r, q); };
            for (int p = 0; p < 2; ++p) {
                for (int m = 0; m < 2; ++m) {
                    c64[t].a[p][m] = 0.5 * (M(p, m) - M(p, 4 - m));
                    c64[t].b[p][m] = 0.5 * (M(p, m) + M(p, 4 - m));
                }
                c64[t].g[p] = M(p, 2);
                c64[t].d[p] = M(2, p);
            }
        }
        const int ok = asym <= 1e-12 * hmax ? 1 : 0;
        // S = D^T diag(w) D of the one-contraction lines, w the GLL weights of 5 points; its rows
        // sum to zero, but for what rounding leaves, when constants have no derivative (sum_k H(k, p) = 0)
        const double gw[5] = {0.1, 49.0 / 90.0, 32.0 / 45.0, 49.0 / 90.0, 0.1};
        double rows = 0.0;
        for (int p = 0; p < 5; ++p) {
            double t = 0.0;
            for (int k = 0; k < 5; ++k) t += D1(p, k);
            rows = std::max(rows, std::fabs(t));
        }
        uni = ok && rows <= 8 * 2.2e-16 * hmax;   // rounding of H only
        UniCoef u;
        auto S = [&](int i, int k) {
            long double t = 0.0L;
            for (int p = 0; p < 5; ++p) t += (long double)D2(i, p) * gw[p] * D1(p, k);
            return t;
        };
        for (int p = 0; p < 2; ++p) {
            for (int m = 0; m < 2; ++m) {
                u.a[p][m] = (double)(0.5L * (S(p, m) - S(p, 4 - m)));
                u.b[p][m] = (double)(0.5L * (S(p, m) + S(p, 4 - m)));
            }
            u.d[p] = (double)S(2, p);
        }
        {   // b g = the row sums of rows 0 and 1; row 2's follows, since they add up to (D 1)^T w (D 1), 1e-30
            const double b00 = u.b[0][0], b01 = u.b[0][1], b10 = u.b[1][0], b11 = u.b[1][1], det = b00 * b11 - b01 * b10;
            auto rho = [&](int p) { return (double)(S(p, 0) + S(p, 1) + S(p, 2) + S(p, 3) + S(p, 4)); };
            u.g[0] = uni ? (b11 * rho(0) - b01 * rho(1)) / det : 0.0;
            u.g[1] = uni ? (b00 * rho(1) - b10 * rho(0)) / det : 0.0;
        }
        for (int p = 0; p < 5; ++p) u.w[p] = gw[p];
        EQC_CUDA(cudaMemcpyToSymbolAsync(cUni, &u, sizeof(u), 0, cudaMemcpyHostToDevice, s));
        EQC_CUDA(cudaMemcpyToSymbolAsync(cEO, c, sizeof(c), 0, cudaMemcpyHostToDevice, s));
        EQC_CUDA(cudaMemcpyToSymbolAsync(cEO64, c64, sizeof(c64), 0, cudaMemcpyHostToDevice, s));
        EQC_CUDA(cudaMemcpyToSymbolAsync(cEO_ok, &ok, sizeof(int), 0, cudaMemcpyHostToDevice, s));
    }
    EQC_CUDA(cudaStreamSynchronize(s));
    // kernel attributes are set here, at handle creation, never during a stream capture
    g_pipe_blocks[0] = resident_blocks(k_apply_pipe<float, LTEX, LTEY, LNT>, LNT, PipeLayout<float, LTEX, LTEY>::BYTES);
    g_pipe_blocks[1] = resident_blocks(k_apply_pipe<double, LTEX, LTEY, LNT>, LNT, PipeLayout<double, LTEX, LTEY>::BYTES);
    uni_setup();
    g_walk_slots = resident_blocks(k_apply_walk, 32 * WK_ROWS, WK_BYTES);
    return uni;
}

// Element-per-lane apply: variant 0 -> 6 element rows per CTA (default), 4..7 -> 4, 6, 8, 12.
static void launch_rows(const float* x, float* y, const ApplyArgs<float>& A, float sign, int zr, cudaStream_t s,
                        const OpEpi<float>& E = OpEpi<float>()) {
    const int sx = (A.L.NelX + 1 + 30) / 31;
    auto go = [&](auto rows_tag, auto minb_tag) {
        constexpr int R = decltype(rows_tag)::value, M = decltype(minb_tag)::value;
        dim3 g(sx, (A.L.NelY + 1 + R - 1) / R);
        k_apply_rows<R, M><<<g, 32 * (R + 1), 0, s>>>(x, y, A, sign, zr, E);
    };
    using I = std::integral_constant<int, 0>;
    (void)sizeof(I);
    switch (A.variant) {
        case 4: go(std::integral_constant<int, 4>{}, std::integral_constant<int, 3>{}); break;
        case 5: go(std::integral_constant<int, 8>{}, std::integral_constant<int, 2>{}); break;
        case 6: go(std::integral_constant<int, 12>{}, std::integral_constant<int, 1>{}); break;
        case 7: go(std::integral_constant<int, 6>{}, std::integral_constant<int, 2>{}); break;
        default: go(std::integral_constant<int, 6>{}, std::integral_constant<int, 3>{}); break;
    }
    EQC_CHECK_LAUNCH();
    count_launch();
}

template <class T>
void apply_K(const T* x, T* y, const ApplyArgs<T>& A, T sign, int mode, cudaStream_t s) {
    if (mode <= 1) {
        dim3 grid(A.L.NelX / LTEX + 1, A.L.NelY / LTEY + 1);
        if constexpr (sizeof(T) == 4) {
            if (A.variant == 8 && A.Wp && aligned16(x) && aligned16(y) && launch_walk(x, y, A, sign, mode == 1 ? 1 : 0, s))
                return;
            if ((A.variant == 0 || A.variant >= 4) && A.Wp && aligned16(x) && aligned16(y)) {
                launch_rows(x, y, A, sign, mode == 1 ? 1 : 0, s);
                return;
            }
        }
        if constexpr (sizeof(T) == 8) {
            const CUtensorMap* uu = (A.uni && A.tma && (A.variant == 0 || A.variant > 3)) ? tma_umap_uni(*A.tma, x, A.L) : nullptr;
            if (uu) {
                launch_uni64(*uu, y, A, sign, mode == 1 ? 1 : 0, s);
                return;
            }
        }
        const CUtensorMap* um = (A.tma && A.variant != 2) ? tma_umap<T>(*A.tma, x, A.L) : nullptr;
        if (um && A.variant == 1) {
            k_apply_tma<T, LTEX, LTEY, LNT><<<grid, LNT, 0, s>>>(*um, tma_wmap<T>(*A.tma), y, A, sign, mode == 1 ? 1 : 0);
        } else if (um) {
            const int ntx = (int)grid.x, ntiles = (int)(grid.x * grid.y);
            k_apply_pipe<T, LTEX, LTEY, LNT><<<std::min(ntiles, pipe_blocks<T>()), LNT, PipeLayout<T, LTEX, LTEY>::BYTES, s>>>(
                *um, tma_wmap<T>(*A.tma), y, A, sign, mode == 1 ? 1 : 0, ntx, ntiles);
        } else {
            k_apply_lines<T, LTEX, LTEY, LNT><<<grid, LNT, 0, s>>>(x, y, A, sign, mode == 1 ? 1 : 0);
        }
        EQC_CHECK_LAUNCH();
        count_launch();
        return;
    }
    const int grid = (A.L.NelX + STX - 1) / STX;
    if (mode == 2) k_strip<T, 2><<<grid, ST_THREADS, 0, s>>>(x, y, A, sign);
    else k_strip<T, 3><<<grid, ST_THREADS, 0, s>>>(x, y, A, sign);
    EQC_CHECK_LAUNCH();
    count_launch();
}

bool apply_K_fault32(const float* x, float* y, const ApplyArgs<float>& A, cudaStream_t s) {
    if (!A.Wp || !aligned16(x) || !aligned16(y)) return false;
    // one element row per CTA (warp 0 the virtual row below the fault, W = 0), grid row 0 only
    const dim3 g((A.L.NelX + 1 + 30) / 31, 1);
    k_apply_rows<1, 8><<<g, 64, 0, s>>>(x, y, A, 1.0f, 0, OpEpi<float>());
    EQC_CHECK_LAUNCH();
    count_launch();
    return true;
}

bool apply_K_epi(const float* x, const ApplyArgs<float>& A, int mode, const OpEpi<float>& E, cudaStream_t s) {
    if (mode > 1 || !A.Wp || !aligned16(x)) return false;
    if (A.variant == 8 && launch_walk(x, nullptr, A, 1.0f, mode, s, E)) return true;
    if (A.variant == 0 || (A.variant >= 4 && A.variant <= 7)) {
        launch_rows(x, nullptr, A, 1.0f, mode, s, E);
        return true;
    }
    return false;
}

bool apply_K_epi(const double* x, const ApplyArgs<double>& A, int mode, const OpEpi<double>& E, cudaStream_t s) {
    if (mode > 1 || !A.uni || !A.tma || (A.variant >= 1 && A.variant <= 3)) return false;
    const CUtensorMap* uu = tma_umap_uni(*A.tma, x, A.L);
    if (!uu) return false;
    launch_uni64(*uu, nullptr, A, 1.0, mode, s, E);
    return true;
}

bool apply_K_dot(const double* x, double* y, const ApplyArgs<double>& A, const DotOut& dot, cudaStream_t s) {
    if (!A.uni || !A.tma || (A.variant >= 1 && A.variant <= 3)) return false;
    const CUtensorMap* uu = tma_umap_uni(*A.tma, x, A.L);
    if (!uu) return false;
    OpEpi<double> E;
    E.x = x;
    launch_uni64(*uu, y, A, 1.0, 1, s, E, dot);
    return true;
}

bool apply_K_residual(const double* x, const ApplyArgs<double>& A, const ResidualOut& R, cudaStream_t s) {
    if (!A.uni || !A.tma || (A.variant >= 1 && A.variant <= 3)) return false;
    const CUtensorMap* uu = tma_umap_uni(*A.tma, x, A.L);
    if (!uu) return false;
    launch_uni64(*uu, nullptr, A, -1.0, 1, s, OpEpi<double>(), R);
    return true;
}

template void apply_K<double>(const double*, double*, const ApplyArgs<double>&, double, int, cudaStream_t);
template void apply_K<float>(const float*, float*, const ApplyArgs<float>&, float, int, cudaStream_t);

}  // namespace eqc
