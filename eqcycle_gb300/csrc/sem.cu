// FP32 stiffness operator of the quasi-static solve, one lane per element, for models whose elements
// have one rigidity each (Handle::mu32, classify_elements).
//
// A line of such an element is one contraction with S = D^T diag(w) D scaled by c mu w_j (see
// kapply.cu's UniCoef; the same form in FP32): 256 operations per element where the two contractions
// with W between them take 560, and four bytes of element data where W takes 112.  A warp whose
// elements include one of several rigidities reads their W and takes both contractions.
//
// A warp owns a strip of 31 element columns (lane 0 is the column left of them) and walks up `rows`
// element rows, keeping the top node row and the top-row contributions of the row below in
// registers; it starts one row early for those contributions.  No shared memory, no barrier: a warp's
// loads of the next row are in flight while it computes.  Every warp is independent, so small
// meshes spread over as many SMs as they have strip rows and large ones run as one wave.
#include "sem.h"
#include "reduce.cuh"
#include "vec.cuh"
#include "cg.cuh"
#include <algorithm>
#include <cmath>

namespace eqc {

// rho: the row sums, which vanish but for the rounding of the two contractions' coefficients (1.6e-7).  They
// stay in so that an element has one operator in either form, to 1e-8 on smooth fields (set_H_sem): CG stops
// at the error that this operator's difference from the FP64 one leaves, 2e-9 of |d| on 480 x 960 elements
// at a tolerance of 1e-10, and a second operator stops 1.5e-9 away from it.
struct UniCoefF {
    float a[2][2], b[2][2], d[2], rho[3];
};
struct EOCoefF {
    float a[2][2], b[2][2], g[2], d[2];
};
__constant__ UniCoefF cUniF;
__constant__ EOCoefF cEOF[2];

__device__ __forceinline__ void uni_line(const float (&v)[5], float (&s)[5]) {
    const float o0 = v[0] - v[4], o1 = v[1] - v[3];
    const float e0 = fmaf(2.f, v[4] - v[2], o0), e1 = fmaf(2.f, v[3] - v[2], o1);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const float P = fmaf(cUniF.a[p][1], o1, cUniF.a[p][0] * o0);
        const float Q = fmaf(cUniF.rho[p], v[2], fmaf(cUniF.b[p][1], e1, cUniF.b[p][0] * e0));
        s[p] = Q + P;
        s[4 - p] = Q - P;
    }
    s[2] = fmaf(cUniF.rho[2], v[2], fmaf(cUniF.d[1], e1, cUniF.d[0] * e0));
}
__device__ __forceinline__ void eo_line(const float (&v)[5], float (&s)[5], const EOCoefF& c) {
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

// Element data and geometry of a launch.
struct SemGeom {
    Layout L;
    const float *mu, *Wp;
    float cx[3], cy[3];   // c1 w_j, c2 w_i, times the unit of mu and the scale of the coefficients
    float c1, c2;
    int rows, ldc;
};

constexpr unsigned FULL = 0xffffffffu;

// The contributions of one element: own nodes out[j][i] (i, j < 4), right column R[j], top row T[i].
__device__ __forceinline__ void element_lines(const float (&u)[5][5], float mu, const float* __restrict__ Wp, bool real,
                                              const SemGeom& G, float (&out)[4][4], float (&R)[4], float (&T)[5]) {
    if (__all_sync(FULL, mu >= 0.f)) {
        const float kx[5] = {mu * G.cx[0], mu * G.cx[1], mu * G.cx[2], mu * G.cx[1], mu * G.cx[0]};
        const float ky[5] = {mu * G.cy[0], mu * G.cy[1], mu * G.cy[2], mu * G.cy[1], mu * G.cy[0]};
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            float s[5];
            uni_line(u[j], s);
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                if (j == 4) T[i] = kx[j] * s[i];
                else if (i == 4) R[j] = kx[j] * s[i];
                else out[j][i] = kx[j] * s[i];
            }
        }
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const float v[5] = {u[0][i], u[1][i], u[2][i], u[3][i], u[4][i]};
            float s[5];
            uni_line(v, s);
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                if (j == 4) T[i] = fmaf(ky[i], s[j], T[i]);
                else if (i == 4) R[j] = fmaf(ky[i], s[j], R[j]);
                else out[j][i] = fmaf(ky[i], s[j], out[j][i]);
            }
        }
        return;
    }
    auto W = [&](int q) { return real ? __ldg(Wp + q) : 0.f; };
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        float s[5], o[5];
        eo_line(u[j], s, cEOF[0]);
#pragma unroll
        for (int p = 0; p < 5; ++p) s[p] *= W(p + 5 * j);
        eo_line(s, o, cEOF[1]);
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            if (j == 4) T[i] = G.c1 * o[i];
            else if (i == 4) R[j] = G.c1 * o[i];
            else out[j][i] = G.c1 * o[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const float v[5] = {u[0][i], u[1][i], u[2][i], u[3][i], u[4][i]};
        float s[5], o[5];
        eo_line(v, s, cEOF[0]);
#pragma unroll
        for (int p = 0; p < 5; ++p) s[p] *= W(i + 5 * p);
        eo_line(s, o, cEOF[1]);
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            if (j == 4) T[i] = fmaf(G.c2, o[j], T[i]);
            else if (i == 4) R[j] = fmaf(G.c2, o[j], R[j]);
            else out[j][i] = fmaf(G.c2, o[j], out[j][i]);
        }
    }
}

__device__ __forceinline__ float4 f4(float v) { return make_float4(v, v, v, v); }
__device__ __forceinline__ float at(const float4& v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w)); }

// WARPS warps per CTA, stacked upwards; grid (strips, groups of WARPS * G.rows element rows).
// Loads are not predicated: indices are clamped into the grid, since an element outside the mesh has
// rigidity 0 and what its lane or row reads does not count.  Offsets are 32-bit byte offsets from the
// vectors' uniform base addresses.
template <int LOAD, int EPI, int PREV, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 16 / WARPS) k_sem(SemGeom G, SemOp O) {
    const Layout L = G.L;
    const int lane = threadIdx.x & 31;
    const int wid = WARPS == 1 ? 0 : __shfl_sync(FULL, (int)(threadIdx.x >> 5), 0);
    const int ex = 31 * (int)blockIdx.x - 1 + lane;
    const int r0 = ((int)blockIdx.y * WARPS + wid) * G.rows;
    const int r1 = min(r0 + G.rows, L.NelY + 1);   // element row NelY is the virtual top row
    const bool own = ex >= 0 && ex <= L.NelX && lane > 0;
    const bool inner = ex >= 0 && ex < L.NelX;     // a real element's column
    const unsigned ld4 = 4u * L.ld, lo = 16u * min(max(ex, 0), L.NelX), lo4 = 16u * min(max(ex + 1, 0), L.NelX);
    auto row_off = [&](int iy) { return (unsigned)min(max(iy, 0), L.ny - 1) * ld4; };
    auto ld16 = [](const float* p, unsigned off) {
        return __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const char*>(p) + off));
    };
    auto ld4b = [](const float* p, unsigned off) {
        return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + off));
    };
    auto st16 = [](float* p, unsigned off, const float4& v) {
        *reinterpret_cast<float4*>(reinterpret_cast<char*>(p) + off) = v;
    };
    // constant element data before the wait for the launches this one depends on
    const unsigned mo = 4u * min(max(ex, 0), L.NelX - 1);
    auto mu_at = [&](int er) {
        const float m = ld4b(G.mu, (unsigned)min(max(er, 0), L.NelY - 1) * (4u * L.NelX) + mo);
        return inner && er >= 0 && er < L.NelY ? m : 0.f;
    };
    float mu = mu_at(r0 - 1), mu_next = mu_at(r0);
    EQC_GRID_WAIT();
    const float *va = LOAD == SL_FIRST ? O.b : O.x, *vb = O.dinv;
    float *pnew = O.uout, beta = 0.f;
    if constexpr (LOAD == SL_DIR) {
        const bool odd = O.S->it & 1;
        vb = odd ? O.p0 : O.p1;
        pnew = odd ? O.p1 : O.p0;
        beta = O.S->restart ? 0.f : O.S->beta32;
    }
    DotAcc<float> acc;

    // raw loads of node row iy: the lane's 4 nodes and the one right of them, of one or two vectors
    struct Raw {
        float4 a, b;
        float a4, b4;
    };
    auto load_row = [&](int iy) {
        Raw w;
        const unsigned row = row_off(iy);
        w.a = ld16(va, row + lo);
        w.a4 = ld4b(va, row + lo4);
        if constexpr (LOAD == SL_FIRST || LOAD == SL_DIR) {
            w.b = ld16(vb, row + lo);
            w.b4 = ld4b(vb, row + lo4);
        }
        return w;
    };
    // coarse values of vertex row vy at the element's two vertex columns
    auto load_xc = [&](int vy) {
        const unsigned row = (unsigned)min(max(vy, 0), L.NelY) * (4u * G.ldc);
        return make_float2(ld4b(O.xc, row + (lo >> 2)), ld4b(O.xc, row + (lo4 >> 2)));
    };
    float2 cl = make_float2(0.f, 0.f), ch = cl;   // vertex rows er and er + 1
    // node row j of element row er from its raw loads
    auto form_row = [&](const Raw& w, int j, float (&u)[5]) {
        u[0] = w.a.x;
        u[1] = w.a.y;
        u[2] = w.a.z;
        u[3] = w.a.w;
        u[4] = w.a4;
        if constexpr (LOAD == SL_FIRST || LOAD == SL_DIR) {
            const float b[5] = {w.b.x, w.b.y, w.b.z, w.b.w, w.b4};
#pragma unroll
            for (int i = 0; i < 5; ++i)
                u[i] = LOAD == SL_FIRST ? cheb_first_pt(b[i], u[i], O.inv_theta) : __fmaf_rn(beta, b[i], u[i]);
        } else if constexpr (LOAD == SL_PROLONG) {
            const float a0 = j == 4 ? ch.x : gll_interp(O.w, j & 3, cl.x, ch.x);
            const float a1 = j == 4 ? ch.y : gll_interp(O.w, j & 3, cl.y, ch.y);
            u[0] = __fadd_rn(u[0], a0);
            u[4] = __fadd_rn(u[4], a1);
#pragma unroll
            for (int i = 1; i < 4; ++i) u[i] = inner ? __fadd_rn(u[i], gll_interp(O.w, i, a0, a1)) : 0.f;   // else padding
        }
    };

    float u[5][5], T[5];
    float S01 = 0.f, S11 = 0.f;   // SE_RESTRICT: the row below's share of this row's vertices
    {
        Raw w[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) w[j] = load_row(4 * (r0 - 1) + j);
        if constexpr (LOAD == SL_PROLONG) {
            cl = load_xc(r0 - 1);
            ch = load_xc(r0);
        }
#pragma unroll
        for (int j = 0; j < 5; ++j) form_row(w[j], j, u[j]);
    }
    auto residual_sums = [&](const float4 (&bv)[4], const float (&out)[4][4], int er, float (&Lx)[4], float (&Hx)[4]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool ok = ex >= 0 && ex <= L.NelX && 4 * er + j >= 1 && 4 * er + j < L.ny;
            float r[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] = ok && (i == 0 || inner) ? __fsub_rn(at(bv[j], i), out[j][i]) : 0.f;
            Lx[j] = restrict_lo(O.w, r[0], r[1], r[2], r[3]);
            Hx[j] = restrict_hi(O.w, r[1], r[2], r[3]);
        }
        S01 = restrict_hi(O.w, Lx[1], Lx[2], Lx[3]);
        S11 = restrict_hi(O.w, Hx[1], Hx[2], Hx[3]);
    };
    {   // the row below the walk: its top-row contributions, and for the restriction its residual's sums
        const int er = r0 - 1;
        float out[4][4], R[4];
        float4 bv[4];
        if constexpr (EPI == SE_RESTRICT) {
#pragma unroll
            for (int j = 0; j < 4; ++j) bv[j] = ld16(O.b, row_off(4 * er + j) + lo);
        }
        element_lines(u, mu, G.Wp + ((int64_t)er * L.NelX + ex) * 28, inner && er >= 0 && er < L.NelY, G, out, R, T);
        if constexpr (EPI == SE_RESTRICT) {   // (its own bottom row is not asked for)
#pragma unroll
            for (int j = 1; j < 4; ++j) out[j][0] += __shfl_up_sync(FULL, R[j], 1);
            float Lx[4], Hx[4];
            residual_sums(bv, out, er, Lx, Hx);
        }
        mu = mu_next;
        mu_next = mu_at(r0 + 1);
    }
    for (int er = r0; er < r1; ++er) {
        unsigned off[4];   // the owned nodes of rows 4 er + j
#pragma unroll
        for (int j = 0; j < 4; ++j) off[j] = row_off(4 * er + j) + lo;
        {
            Raw w[4];
#pragma unroll
            for (int j = 1; j < 5; ++j) w[j - 1] = load_row(4 * er + j);
            if constexpr (LOAD == SL_PROLONG) {
                cl = ch;
                ch = load_xc(er + 1);
            }
#pragma unroll
            for (int i = 0; i < 5; ++i) u[0][i] = u[4][i];
#pragma unroll
            for (int j = 1; j < 5; ++j) form_row(w[j - 1], j, u[j]);
        }
        // this row's epilogue operands, in flight during the lines
        float4 bv[4], dv[4], pv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if constexpr (EPI != SE_STORE) bv[j] = ld16(O.b, off[j]);
            if constexpr (EPI == SE_CHEB) dv[j] = ld16(O.dinv, off[j]);
            if constexpr (PREV == SP_VEC)   // written in place: a plain load
                pv[j] = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(O.xp) + off[j]);
        }
        float out[4][4], R[4], Tn[5];
        element_lines(u, mu, G.Wp + ((int64_t)er * L.NelX + ex) * 28, inner && er < L.NelY, G, out, R, Tn);
        mu = mu_next;
        mu_next = mu_at(er + 2);
        // contributions of the left element (right column) and of the element row below (top row)
#pragma unroll
        for (int j = 0; j < 4; ++j) out[j][0] += __shfl_up_sync(FULL, R[j], 1);
        const float T4 = __shfl_up_sync(FULL, T[4], 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) out[0][i] += T[i];
        out[0][0] += T4;
#pragma unroll
        for (int i = 0; i < 5; ++i) T[i] = Tn[i];
        if (er == 0) {   // the fault row is not part of the system
#pragma unroll
            for (int i = 0; i < 4; ++i) out[0][i] = 0.f;
        }
        if constexpr (EPI == SE_RESTRICT) {
            const float S01b = S01, S11b = __shfl_up_sync(FULL, S11, 1);
            float Lx[4], Hx[4];
            residual_sums(bv, out, er, Lx, Hx);
            const float S00 = restrict_lo(O.w, Lx[0], Lx[1], Lx[2], Lx[3]);
            const float S10 = __shfl_up_sync(FULL, restrict_lo(O.w, Hx[0], Hx[1], Hx[2], Hx[3]), 1);
            if (own) {
                const float v = er >= 1 ? restrict_sum(S00, S10, S01b, S11b) : 0.f;
                const int64_t o = (int64_t)er * G.ldc + ex;
                O.bc[o] = v;
                cheb_first_store(O.first, o, v);
            }
        } else if (own) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j > 0 && er == L.NelY) break;   // the virtual row has one node row
                float4 t = make_float4(out[j][0], out[j][1], out[j][2], out[j][3]);
                const float4 uo = make_float4(u[j][0], u[j][1], u[j][2], u[j][3]);
                if constexpr (LOAD == SL_PROLONG || LOAD == SL_DIR) st16(pnew, off[j], uo);
                if constexpr (EPI == SE_CHEB) {
                    float4 up = uo;
                    if constexpr (PREV == SP_VEC) up = pv[j];
                    if constexpr (PREV == SP_ZERO) up = f4(0.f);
                    if constexpr (PREV == SP_FIRST)
                        up = make_float4(cheb_first_pt(dv[j].x, bv[j].x, O.inv_theta), cheb_first_pt(dv[j].y, bv[j].y, O.inv_theta),
                                         cheb_first_pt(dv[j].z, bv[j].z, O.inv_theta), cheb_first_pt(dv[j].w, bv[j].w, O.inv_theta));
                    t = make_float4(cheb_x_pt(uo.x, up.x, bv[j].x, t.x, dv[j].x, O.c1, O.c2),
                                    cheb_x_pt(uo.y, up.y, bv[j].y, t.y, dv[j].y, O.c1, O.c2),
                                    cheb_x_pt(uo.z, up.z, bv[j].z, t.z, dv[j].z, O.c1, O.c2),
                                    cheb_x_pt(uo.w, up.w, bv[j].w, t.w, dv[j].w, O.c1, O.c2));
                }
                st16(O.out, off[j], t);
                if constexpr (WARPS > 1) {
                    const float4 v = EPI == SE_CHEB ? bv[j] : uo;
                    acc.add(t.x, v.x);
                    acc.add(t.y, v.y);
                    acc.add(t.z, v.z);
                    acc.add(t.w, v.w);
                }
            }
        }
    }
    if constexpr (WARPS > 1) {
        grid_sum(acc, O.part, O.count, [&](double t) { cg_take_dot(O.S, t, O.dot == 2); });
    }
}

// c w_j in FP32, each remainder carried into the next smaller one: 2 + 2 + 1 of them sum to 2 c within 4e-9,
// where each rounded by itself would scale the operator by up to 3e-8.
static void line_weights(double c, float* out) {
    const double w[3] = {0.1 * c, 49.0 / 90.0 * c, 32.0 / 45.0 * c};
    out[2] = (float)w[2];
    const double t = w[1] + 0.5 * (w[2] - out[2]);
    out[1] = (float)t;
    out[0] = (float)(w[0] + (t - out[1]));
}

bool sem_usable(const Handle& h) { return h.sem_ok && h.opt.apply_variant == 0; }

void sem_launch(Handle& h, SemLoad load, SemEpi epi, SemPrev prev, const SemOp& o) {
    const Layout& L = h.L;
    SemGeom G;
    G.L = L;
    G.mu = h.mu32.p;
    G.Wp = h.W32p.p;
    G.c1 = (float)h.c1;
    G.c2 = (float)h.c2;
    line_weights(h.c1 * h.mu_unit * h.sem_scale, G.cx);
    line_weights(h.c2 * h.mu_unit * h.sem_scale, G.cy);
    G.ldc = L.NelX + 1;
    const int nsx = (L.NelX + 1 + 30) / 31;
    // rows per warp: the fewest with which every warp is resident at once (16 on each of 152 SMs; ms per step on
    // 480 x 960 elements 7.13, and 8.19, 7.78 and 7.59 with the rows for 8, 24 and 40)
    const int64_t warps = (int64_t)nsx * (L.NelY + 1), slots = 152 * 16;
    G.rows = (int)((warps + slots - 1) / slots);
    // a sum's end is per CTA: eight warps to one (ms per step on 240 x 480 elements 2.70 with four, 2.66 with eight, on
    // 480 x 960 7.45 and 7.43, the same on 48 x 48)
    const int W = o.dot ? 8 : 1;
    const dim3 grid(nsx, (L.NelY + W * G.rows) / (W * G.rows));
    auto go = [&](auto kernel) { kernel<<<grid, 32 * W, 0, h.stream>>>(G, o); };
    const bool dot = o.dot != 0;
    if (load == SL_PLAIN && epi == SE_STORE && !dot) go(k_sem<SL_PLAIN, SE_STORE, SP_NONE, 1>);
    else if (load == SL_DIR && epi == SE_STORE && dot) go(k_sem<SL_DIR, SE_STORE, SP_NONE, 8>);
    else if (load == SL_PLAIN && epi == SE_RESTRICT && !dot) go(k_sem<SL_PLAIN, SE_RESTRICT, SP_NONE, 1>);
    else if (load == SL_FIRST && epi == SE_CHEB && prev == SP_ZERO && !dot) go(k_sem<SL_FIRST, SE_CHEB, SP_ZERO, 1>);
    else if (load == SL_PLAIN && epi == SE_CHEB && prev == SP_FIRST && !dot) go(k_sem<SL_PLAIN, SE_CHEB, SP_FIRST, 1>);
    else if (load == SL_PLAIN && epi == SE_CHEB && prev == SP_VEC && !dot) go(k_sem<SL_PLAIN, SE_CHEB, SP_VEC, 1>);
    else if (load == SL_PLAIN && epi == SE_CHEB && prev == SP_VEC) go(k_sem<SL_PLAIN, SE_CHEB, SP_VEC, 8>);
    else if (load == SL_PROLONG && epi == SE_CHEB && prev == SP_NONE && !dot) go(k_sem<SL_PROLONG, SE_CHEB, SP_NONE, 1>);
    else if (load == SL_PROLONG && epi == SE_CHEB && prev == SP_NONE) go(k_sem<SL_PROLONG, SE_CHEB, SP_NONE, 8>);
    else throw Error(EQC_E_STATE, "spectral-element operator: no such combination");
    EQC_CHECK_LAUNCH();
    count_launch();
}

// S = D2 diag(w) D1 with D1 and D2 the two contractions as their FP32 coefficients have them.  Its entries
// are rounded once more; the scale that gives a linear field's energy back goes into the lines' weights.
double set_H_sem(const double* H, cudaStream_t s) {
    const double gw[5] = {0.1, 49.0 / 90.0, 32.0 / 45.0, 49.0 / 90.0, 0.1};
    EOCoefF c[2];
    double D[2][5][5];
    for (int t = 0; t < 2; ++t) {
        auto M = [&](int r, int q) { return t == 0 ? H[q + 5 * r] : H[r + 5 * q]; };
        for (int p = 0; p < 2; ++p) {
            for (int m = 0; m < 2; ++m) {
                const double a = c[t].a[p][m] = (float)(0.5 * (M(p, m) - M(p, 4 - m)));
                const double b = c[t].b[p][m] = (float)(0.5 * (M(p, m) + M(p, 4 - m)));
                D[t][p][m] = a + b;
                D[t][p][4 - m] = b - a;
                D[t][4 - p][m] = a - b;
                D[t][4 - p][4 - m] = -a - b;
            }
            D[t][p][2] = c[t].g[p] = (float)M(p, 2);
            D[t][4 - p][2] = -D[t][p][2];
            D[t][2][p] = c[t].d[p] = (float)M(2, p);
            D[t][2][4 - p] = -D[t][2][p];
        }
        D[t][2][2] = 0.0;
    }
    auto S = [&](int i, int k) {
        long double t = 0.0L;
        for (int p = 0; p < 5; ++p) t += (long double)D[1][i][p] * gw[p] * D[0][p][k];
        return t;
    };
    UniCoefF u;
    const double xi[2] = {1.0, std::sqrt(3.0 / 7.0)};
    double exact = 0.0, rounded = 0.0;
    for (int p = 0; p < 2; ++p) {
        for (int m = 0; m < 2; ++m) {
            const double a = (double)(0.5L * (S(p, m) - S(p, 4 - m)));
            u.a[p][m] = (float)a;
            u.b[p][m] = (float)(0.5L * (S(p, m) + S(p, 4 - m)));
            exact += xi[p] * xi[m] * a;
            rounded += xi[p] * xi[m] * u.a[p][m];
        }
        u.d[p] = (float)S(2, p);
    }
    for (int p = 0; p < 3; ++p) u.rho[p] = (float)(S(p, 0) + S(p, 1) + S(p, 2) + S(p, 3) + S(p, 4));
    EQC_CUDA(cudaMemcpyToSymbolAsync(cUniF, &u, sizeof(u), 0, cudaMemcpyHostToDevice, s));
    EQC_CUDA(cudaMemcpyToSymbolAsync(cEOF, c, sizeof(c), 0, cudaMemcpyHostToDevice, s));
    EQC_CUDA(cudaStreamSynchronize(s));
    return rounded > 0.0 && exact > 0.0 ? exact / rounded : 1.0;
}

}  // namespace eqc
