// K1 in double-float: y = sign * K x for FP64 x and y, evaluated with FP32 operations on
// unevaluated hi + lo pairs (df.cuh), ~1e-14 relative per operation, for callers that need an
// FP64-class apply at the FP32 rate (eqc_apply_K_device dtype 2, and the mixed solver's
// intermediate reliable updates, r -= K dx with dx the correction since the previous update).
// The solver's full true residuals b - K_II x do not use it: late in a cycle the displacement
// grows until the 1e-14 error of K x floors the residual near 1e-5 of |b|, above the CG
// tolerance (measured), so those stay FP64; K dx has the size of the residual it corrects.
//
// Bound by FP32 issue on large meshes (127 us on 480 x 960 elements, 39 on 240 x 480; with both
// contractions of every line 236 and 64) and by one CTA's instruction chain, 27 us, on small ones, where
// the FP64 apply takes its place (df_pays).
// With ResidualOut the launch applies the change to the residual and takes its norm: no K dx array, no pass
// over it afterwards.
//
// Layout as k_apply_rows: one lane per element, one warp per element row of 31 elements plus a
// halo lane, ROWS element rows per CTA plus a halo warp; the line contractions in even-odd form.
// Where every element of a warp has one rigidity (Handle::mu64) a line is one contraction (kapply.cu's
// UniCoef), 235 FP32 operations instead of 533; otherwise both contractions with W between them, each
// lane reading its element's nodes twice (rows for the x-lines, columns for the y-lines; L1 hits).
#include "model.h"
#include "df.cuh"
#include "cg.cuh"
#include <cmath>

namespace eqc {

struct EODF {
    df a[2][2], b[2][2], g[2], d[2];
};
__constant__ EODF cEOdf[2];   // [0]: s_p = sum_k H(k,p) v_k ; [1]: o_i = sum_p H(i,p) s_p

__device__ __forceinline__ void eo5_df(const df (&v)[5], df (&s)[5], const EODF& c) {
    const df e0 = df_add(v[0], v[4]), e1 = df_add(v[1], v[3]);
    const df o0 = df_sub(v[0], v[4]), o1 = df_sub(v[1], v[3]);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const df P = df_add(df_mul(c.a[p][0], o0), df_mul(c.a[p][1], o1));
        const df Q = df_add(df_add(df_mul(c.b[p][0], e0), df_mul(c.b[p][1], e1)), df_mul(c.g[p], v[2]));
        s[p] = df_add(P, Q);
        s[4 - p] = df_sub(P, Q);
    }
    s[2] = df_add(df_mul(c.d[0], o0), df_mul(c.d[1], o1));
}

struct UniDF {
    df a[2][2], b[2][2], d[2];
    df cx[3], cy[3];   // c1 w_j, c2 w_i
};
__device__ __forceinline__ df df_twice(df x) { return df{2.f * x.hi, 2.f * x.lo}; }
__device__ __forceinline__ void uni_line_df(const df (&v)[5], df (&s)[5], const UniDF& c) {
    const df o0 = df_sub(v[0], v[4]), o1 = df_sub(v[1], v[3]);
    const df e0 = df_add(df_twice(df_sub(v[4], v[2])), o0), e1 = df_add(df_twice(df_sub(v[3], v[2])), o1);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const df P = df_add(df_mul(c.a[p][0], o0), df_mul(c.a[p][1], o1));
        const df Q = df_add(df_mul(c.b[p][0], e0), df_mul(c.b[p][1], e1));
        s[p] = df_add(Q, P);
        s[4 - p] = df_sub(Q, P);
    }
    s[2] = df_add(df_mul(c.d[0], e0), df_mul(c.d[1], e1));
}

__device__ __forceinline__ df shfl_up_df(df v) {
    return df{__shfl_up_sync(0xffffffffu, v.hi, 1), __shfl_up_sync(0xffffffffu, v.lo, 1)};
}

template <int ROWS, bool RES, bool UNI>
__global__ void __launch_bounds__(32 * (ROWS + 1), 2)
    k_apply_df(const double* __restrict__ x, double* __restrict__ y, const float* __restrict__ Whi,
               const float* __restrict__ Wlo, const double* __restrict__ mu64, int mu_pitch, Layout L, df c1, df c2,
               const __grid_constant__ UniDF U, double sign, int zero_row0, const int* gate, int gate_val, ResidualOut Ro) {
    EQC_GRID_WAIT();
    if (gate && *gate != gate_val) return;
    __shared__ float Th[ROWS + 1][5][32], Tl[ROWS + 1][5][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ex = (int)blockIdx.x * 31 - 1 + lane;
    const int ey = (int)blockIdx.y * ROWS - 1 + w;
    const bool real = ex >= 0 && ex < L.NelX && ey >= 0 && ey < L.NelY;
    const bool halo = w == 0;
    const int64_t eo = real ? ((int64_t)ey * L.NelX + ex) * 28 : 0;
    auto Wd = [&](int q) { return real ? df{__ldg(Whi + eo + q), __ldg(Wlo + eo + q)} : df{0.f, 0.f}; };
    // node (4 ex + i, 4 ey + j) of the element, zero outside the grid
    auto node = [&](int i, int j) {
        const int ix = 4 * ex + i, iy = 4 * ey + j;
        return (ix >= 0 && ix < L.nx && iy >= 0 && iy < L.ny) ? df_from_double_skip(__ldg(x + (int64_t)iy * L.ld + ix))
                                                                  : df{0.f, 0.f};
    };
    const double mu = UNI && real ? __ldg(mu64 + (int64_t)ey * mu_pitch + ex + 1) : 0.0;
    df out[4][4], R[4], T[5];
    if (UNI && __all_sync(0xffffffffu, __double2hiint(mu) >= 0)) {
        const df m = df_from_double(mu);
        // every load before the first conversion; an element outside the mesh reads the nearest one (mu is 0)
        const double* xe = x + (int64_t)(4 * min(max(ey, 0), L.NelY - 1)) * L.ld + 4 * min(max(ex, 0), L.NelX - 1);
        double raw[5][5];
#pragma unroll
        for (int j = 0; j < 5; ++j)
#pragma unroll
            for (int i = 0; i < 5; ++i) raw[j][i] = __ldg(xe + (int64_t)j * L.ld + i);
        df u[5][5];
#pragma unroll
        for (int j = 0; j < 5; ++j)
#pragma unroll
            for (int i = 0; i < 5; ++i) u[j][i] = df_from_double(raw[j][i]);
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            if (halo && j < 4) continue;
            df o[5];
            uni_line_df(u[j], o, U);
            const df k = df_mul(m, U.cx[j < 3 ? j : 4 - j]);
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                const df q = df_mul(k, o[i]);
                if (j == 4) T[i] = q;
                else if (i == 4) R[j] = q;
                else out[j][i] = q;
            }
        }
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const df v[5] = {u[0][i], u[1][i], u[2][i], u[3][i], u[4][i]};
            df o[5];
            uni_line_df(v, o, U);
            const df k = df_mul(m, U.cy[i < 3 ? i : 4 - i]);
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                if (halo && j < 4) continue;
                const df q = df_mul(k, o[j]);
                if (j == 4) T[i] = df_add(T[i], q);
                else if (i == 4) R[j] = df_add(R[j], q);
                else out[j][i] = df_add(out[j][i], q);
            }
        }
    } else {
        // x-lines (the halo warp needs only the top one, for T)
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            if (halo && j < 4) continue;
            df v[5], s[5], o[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] = node(k, j);
            eo5_df(v, s, cEOdf[0]);
#pragma unroll
            for (int p = 0; p < 5; ++p) s[p] = df_mul(s[p], Wd(p + 5 * j));
            eo5_df(s, o, cEOdf[1]);
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                const df q = df_mul(c1, o[i]);
                if (j == 4) T[i] = q;
                else if (i == 4) R[j] = q;
                else out[j][i] = q;
            }
        }
        // y-lines
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            df v[5], s[5], o[5];
#pragma unroll
            for (int l = 0; l < 5; ++l) v[l] = node(i, l);
            eo5_df(v, s, cEOdf[0]);
#pragma unroll
            for (int p = 0; p < 5; ++p) s[p] = df_mul(s[p], Wd(i + 5 * p));
            eo5_df(s, o, cEOdf[1]);
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                if (halo && j < 4) continue;
                const df q = df_mul(c2, o[j]);
                if (j == 4) T[i] = df_add(T[i], q);
                else if (i == 4) R[j] = df_add(R[j], q);
                else out[j][i] = df_add(out[j][i], q);
            }
        }
    }
    if (halo) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int i = 0; i < 4; ++i) out[j][i] = df{0.f, 0.f};
            R[j] = df{0.f, 0.f};
        }
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        Th[w][i][lane] = T[i].hi;
        Tl[w][i][lane] = T[i].lo;
    }
    df Rl[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) Rl[j] = shfl_up_df(R[j]);
    __syncthreads();
    const bool own = !halo && lane > 0 && ex <= L.NelX && ey <= L.NelY;
    DotAcc<float> acc;
    if (own) {
#pragma unroll
        for (int j = 0; j < 4; ++j) out[j][0] = df_add(out[j][0], Rl[j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) out[0][i] = df_add(out[0][i], df{Th[w - 1][i][lane], Tl[w - 1][i][lane]});
        out[0][0] = df_add(out[0][0], df{Th[w - 1][4][lane - 1], Tl[w - 1][4][lane - 1]});
        const double sg = RES ? Ro.S->sigma : 0.0, inv = RES ? Ro.S->inv_sigma : 0.0;
        const int es = RES ? Ro.S->sigma_exp : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int iy = 4 * ey + j;
            if (iy >= L.ny) break;
            const int64_t o = (int64_t)iy * L.ld + 4 * ex;
            if constexpr (RES) {   // r64 -= K dx / sigma off the fault row (the row's padding adds zeros)
                if (iy == 0) continue;
                double r[4];
                float f[4];
                ld4(Ro.r64 + o, r);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    r[i] = __fma_rn(-df_to_double(out[j][i]), inv, r[i]);
                    f[i] = residual32(r[i], es, sg, acc);
                }
                st4(Ro.r64 + o, r);
                st4(Ro.r32 + o, f);
            } else {
                const double z = (zero_row0 && iy == 0) ? 0.0 : sign;
                const double t[4] = {z * df_to_double(out[j][0]), z * df_to_double(out[j][1]), z * df_to_double(out[j][2]),
                                     z * df_to_double(out[j][3])};
                st4(y + o, t);
            }
        }
    }
    if constexpr (RES) residual_done(Ro, acc);
}

static df host_df(double v) {
    const float hi = (float)v;
    return df{hi, (float)(v - (double)hi)};
}

void set_H_df(const double* H, cudaStream_t s) {
    EODF c[2];
    for (int t = 0; t < 2; ++t) {
        auto M = [&](int r, int q) { return t == 0 ? H[q + 5 * r] : H[r + 5 * q]; };
        for (int p = 0; p < 2; ++p) {
            for (int m = 0; m < 2; ++m) {
                c[t].a[p][m] = host_df(0.5 * (M(p, m) - M(p, 4 - m)));
                c[t].b[p][m] = host_df(0.5 * (M(p, m) + M(p, 4 - m)));
            }
            c[t].g[p] = host_df(M(p, 2));
            c[t].d[p] = host_df(M(2, p));
        }
    }
    EQC_CUDA(cudaMemcpyToSymbolAsync(cEOdf, c, sizeof(c), 0, cudaMemcpyHostToDevice, s));
    EQC_CUDA(cudaStreamSynchronize(s));
}

bool apply_K_df(Handle& h, const double* x, double* y, double sign, int mode, cudaStream_t s, const int* gate,
                int gate_val, const ResidualOut* Ro) {
    if (!h.df_ok || mode > 1 || !h.W32lo.p || (reinterpret_cast<uintptr_t>(y) & 15)) return false;
    if (!gate && !Ro && !df_pays(h) && h.opt.apply_variant == 0) {
        apply_K<double>(x, y, args64(h), sign, mode, s);
        return true;
    }
    constexpr int R = DF_ROWS;
    const Layout& L = h.L;
    UniDF U;   // S = D^T diag(w) D in its even-odd form
    const double gw[5] = {0.1, 49.0 / 90.0, 32.0 / 45.0, 49.0 / 90.0, 0.1};
    auto S = [&](int i, int k) {
        long double t = 0.0L;
        for (int p = 0; p < 5; ++p) t += (long double)h.H[i + 5 * p] * gw[p] * h.H[k + 5 * p];
        return t;
    };
    for (int p = 0; p < 2; ++p) {
        for (int m = 0; m < 2; ++m) {
            U.a[p][m] = host_df((double)(0.5L * (S(p, m) - S(p, 4 - m))));
            U.b[p][m] = host_df((double)(0.5L * (S(p, m) + S(p, 4 - m))));
        }
        U.d[p] = host_df((double)S(2, p));
    }
    for (int k = 0; k < 3; ++k) {
        U.cx[k] = host_df(h.c1 * gw[k]);
        U.cy[k] = host_df(h.c2 * gw[k]);
    }
    dim3 g((L.NelX + 1 + 30) / 31, (L.NelY + 1 + R - 1) / R);
    auto go = [&](auto kernel) {
        kernel<<<g, 32 * (R + 1), 0, s>>>(x, y, h.W32p.p, h.W32lo.p, h.mu64.p, mu_pitch(L.NelX), L, host_df(h.c1),
                                          host_df(h.c2), U, sign, mode == 1 ? 1 : 0, gate, gate_val, Ro ? *Ro : ResidualOut());
    };
    if (h.uni_df_pays) {
        if (Ro) go(k_apply_df<R, true, true>);
        else go(k_apply_df<R, false, true>);
    } else {
        if (Ro) go(k_apply_df<R, true, false>);
        else go(k_apply_df<R, false, false>);
    }
    EQC_CHECK_LAUNCH();
    count_launch();
    return true;
}

}  // namespace eqc
