// Learned initial guess: network kernels (forward, backward, Adam), the coarse-grid
// transfers and the time-loop hooks.  See learn.h for the network.
//
// All kernels are deterministic (fixed reduction orders), so training on the same pairs with
// the same seed gives bitwise the same weights.
#include "learn.h"
#include "reduce.cuh"
#include "vec.cuh"
#include "gemm32.cuh"
#include <cmath>
#include <random>
#include <algorithm>

namespace eqc {

__device__ __forceinline__ float tof(float v) { return v; }
__device__ __forceinline__ float tof(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// ---- layers as tiled products (gemm32.cuh) ------------------------------------------------
// What becomes of C(m, n).  sum, sum_done: the row sums of A, where the layer's bias needs them.
struct EpNoSum {
    __device__ void sum(const float (&)[8], int) {}   // of slice t
    __device__ void sum_done(int, int, int) {}
};
struct EpLinear : EpNoSum {   // C = v + bias[n], and its GELU where the next layer takes that
    float* C;
    int64_t ldc;
    const float* bias;
    float* Cg;
    __device__ int64_t npos(int n) const { return n; }
    __device__ void put(int m, int n, int64_t, float v) const {
        v += bias ? bias[n] : 0.f;
        C[m * ldc + n] = v;
        if (Cg) Cg[m * ldc + n] = gelu(v);
    }
};
struct EpGeluGrad : EpNoSum {   // C = v GELU'(z)
    float* C;
    const float* z;
    int64_t ldc;
    __device__ int64_t npos(int n) const { return n; }
    __device__ void put(int m, int n, int64_t, float v) const { C[m * ldc + n] = v * gelu_grad(z[m * ldc + n]); }
};
struct EpConv : EpNoSum {   // n = (b, t), m = channel: z = v + bias[m], a = GELU(z)
    float *z, *a;
    const float* bias;
    int T;
    __device__ int64_t npos(int n) const { return (int64_t)(n / T) * GN_C * T + n % T; }
    __device__ void put(int m, int, int64_t np, float v) const {
        v += bias[m];
        z[np + (int64_t)m * T] = v;
        a[np + (int64_t)m * T] = gelu(v);
    }
};
struct EpConvGrad : EpNoSum {   // n = (b, u) for the positions 2 u + par: g = v GELU'(z)
    float* g;
    const float* z;
    int T, U, par;
    __device__ int64_t npos(int n) const { return (int64_t)(n / U) * GN_C * T + 2 * (n % U) + par; }
    __device__ void put(int m, int, int64_t np, float v) const {
        const int64_t i = np + (int64_t)m * T;
        g[i] = v * gelu_grad(z[i]);
    }
};
// Weight and bias gradients: whole sums (a fully connected layer's K is the batch) or a split's share.  The row
// sums are the first column tile's work, or each column tile's on its slices: every CTA of a split is resident
// at once, so that the longest sets the time (the four layers of 256 pairs: 241 us with all slices summed by one
// tile, 220 now).
template <bool KF, bool PART>
struct EpWeight {
    float* C;
    float* db;         // !PART
    double* db_part;   // PART: [split][column tile][M]
    int M, N;
    RowSum<KF> rs;
    __device__ void sum(const float (&v)[8], int t) {
        if ((PART ? t % gridDim.x : 0) == blockIdx.x) rs.add(v);
    }
    __device__ void sum_done(int m0, int n0, int) {
        if (!PART && n0 != 0) return;
        rs.done(m0, M, [&](int m, double d) {
            if (PART) db_part[((int64_t)blockIdx.z * gridDim.x + blockIdx.x) * M + m] = d;
            else db[m] = (float)d;
        });
    }
    __device__ int64_t npos(int n) const { return (PART ? (int64_t)blockIdx.z * M * N : 0) + n; }
    __device__ void put(int m, int, int64_t np, float v) const { C[np + (int64_t)m * N] = v; }
};
// gW and gb from the splits' shares: 32 results a CTA, every eighth split a warp (481 splits of
// conv1's 640 weights: 73 us with a thread to each result).
__global__ void __launch_bounds__(256) k_weight_sum(const float* __restrict__ part, const double* __restrict__ db_part,
                                                    int splits, int tiles, int M, int N, float* __restrict__ gW,
                                                    float* __restrict__ gb) {
    EQC_GRID_WAIT();
    __shared__ double sh[8][32];
    const int n = M * N, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (i < n) {   // a thread's shares as an error-free pair in FP32: FP64 sums of them took 64 us for 38, with the same bits
        float hi = 0.f, lo = 0.f;
#pragma unroll 8
        for (int z = w; z < splits; z += 8) {
            float t, e;
            two_sum(hi, part[(int64_t)z * n + i], t, e);
            hi = t;
            lo += e;
        }
        s = (double)hi + (double)lo;
    } else if (i < n + M) {
#pragma unroll 8
        for (int z = w; z < splits * tiles; z += 8) s += db_part[(int64_t)z * M + i - n];
    }
    sh[w][lane] = s;
    __syncthreads();
    if (w != 0 || i >= n + M) return;
#pragma unroll
    for (int q = 1; q < 8; ++q) s += sh[q][lane];
    if (i < n) gW[i] = (float)s;
    else gb[i - n] = (float)s;
}

// Convolution operands (kernel 5, stride 2, padding 2).  The layer's input at output position (b, t) and tap
// (ci, k): in[b][ci][2t + k - 2], the positions along mn (forward) or along k (weight gradient).
__device__ __forceinline__ uint32_t raw(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t raw(__nv_bfloat16 v) { return (uint32_t)__bfloat16_as_ushort(v) << 16; }
template <bool KF>
struct OpGather {
    static constexpr bool K_FAST = KF, VEC = false;
    __device__ static float value(const uint32_t (&v)[8], int i) { return __uint_as_float(v[i]); }
};
template <bool POS_K>
struct OpConvIn : OpGather<POS_K> {
    const float* in;
    int Cin, Tin, Tout;
    __device__ TilePtr<float> ptr(int n) const { return {in + (int64_t)(n / Tout) * Cin * Tin, 2 * (n % Tout) - 2}; }
    __device__ TileOff off(int k) const { return {k / GN_K * Tin, k % GN_K}; }
    __device__ uint32_t get(TilePtr<float> a, TileOff b, bool& ok) const {
        const int s = a.s + b.s;
        ok = s >= 0 && s < Tin;
        return raw(a.q[b.off + min(max(s, 0), Tin - 1)]);
    }
};
struct OpConvW : OpGather<true> {   // W[co][ci][k], m = co, k = (ci, k)
    const __nv_bfloat16* W;
    int ld;
    __device__ TilePtr<__nv_bfloat16> ptr(int k) const { return {W + k, 0}; }
    __device__ TileOff off(int m) const { return {m * ld, 0}; }
    __device__ uint32_t get(TilePtr<__nv_bfloat16> a, TileOff b, bool&) const { return raw(a.q[b.off]); }
};
struct OpConvGz : OpGather<true> {   // g_z[b][co][t], m = co, k = (b, t)
    const float* gz;
    int T;
    __device__ TilePtr<float> ptr(int k) const { return {gz + (int64_t)(k / T) * GN_C * T + k % T, 0}; }
    __device__ TileOff off(int m) const { return {m * T, 0}; }
    __device__ uint32_t get(TilePtr<float> a, TileOff b, bool&) const { return raw(a.q[b.off]); }
};
// The input's gradient at s = 2u + par: taps par + 2j, j < J = 3 - par, from the output positions u + 1 - j.
template <int J>
struct OpTapsW : OpGather<false> {   // W[co][m][par + 2j], k = (co, j)
    const __nv_bfloat16* W;
    __device__ TilePtr<__nv_bfloat16> ptr(int m) const { return {W + m * GN_K + 3 - J, 0}; }
    __device__ TileOff off(int k) const { return {k / J * (GN_C * GN_K) + 2 * (k % J), 0}; }
    __device__ uint32_t get(TilePtr<__nv_bfloat16> a, TileOff b, bool&) const { return raw(a.q[b.off]); }
};
template <int J>
struct OpTapsGz : OpGather<false> {   // g_z[b][co][u + 1 - j], n = (b, u)
    const float* gz;
    int T, U;
    __device__ TilePtr<float> ptr(int n) const { return {gz + (int64_t)(n / U) * GN_C * T, n % U + 1}; }
    __device__ TileOff off(int k) const { return {k / J * T, -(k % J)}; }
    __device__ uint32_t get(TilePtr<float> a, TileOff b, bool& ok) const {
        const int t = a.s + b.s;
        ok = t >= 0 && t < T;
        return raw(a.q[b.off + min(max(t, 0), T - 1)]);
    }
};

template <int S, class OA, class OB, class EP>
static void tile_launch(const OA& A, const OB& B, const EP& E, int M, int N, int K, dim3 g, cudaStream_t s) {
    if constexpr (S == 1) {
        k_tile<OA, OB, EP, 1><<<g, GT_THREADS, 0, s>>>(A, B, E, M, N, K, K);
    } else {
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(g.x, g.y, S);
        c.blockDim = dim3(GT_THREADS);
        c.stream = s;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = 1;
        at.val.clusterDim.y = 1;
        at.val.clusterDim.z = S;
        c.attrs = &at;
        c.numAttrs = 1;
        const int chunk = ((K + S - 1) / S + GT_K - 1) / GT_K * GT_K;
        EQC_CUDA(cudaLaunchKernelEx(&c, k_tile<OA, OB, EP, S>, A, B, E, M, N, K, chunk));
    }
    EQC_CHECK_LAUNCH();
    count_launch();
}
// K is split over a cluster where the tiles alone leave SMs idle: up to two CTAs for each SM and 64 of K and
// more to each CTA.  SPLIT: not with row sums, which are of a CTA's K.
template <bool SPLIT = true, class OA, class OB, class EP>
static void tile(const OA& A, const OB& B, const EP& E, int M, int N, int K, cudaStream_t s) {
    if (N == 0) return;   // the odd positions of a layer with one
    const dim3 g((N + GT_N - 1) / GT_N, (M + GT_N - 1) / GT_N);
    const int tiles = (int)(g.x * g.y);
    if constexpr (SPLIT) {
        if (tiles * 8 <= 2 * 152 && K >= 8 * 64) return tile_launch<8>(A, B, E, M, N, K, g, s);
        if (tiles * 4 <= 2 * 152 && K >= 4 * 64) return tile_launch<4>(A, B, E, M, N, K, g, s);
    }
    tile_launch<1>(A, B, E, M, N, K, g, s);
}

// ---- GEMV for small batches (inference): y[b][o] = sum_i x[b][i] W[o][i] + bias[o]; one warp
// per output row o, lanes striding over i in BF16 pairs; optional GELU copy.
template <int BMAX>
__global__ void __launch_bounds__(256) k_gemv(int B, int N, int K, const float* __restrict__ x,
                                              const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias,
                                              float* __restrict__ y, float* __restrict__ yg) {
    EQC_GRID_WAIT();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= N) return;
    const __nv_bfloat16* w = W + (int64_t)warp * K;
    float acc[BMAX];
#pragma unroll
    for (int b = 0; b < BMAX; ++b) acc[b] = 0.f;
    const bool pairs = ((K & 1) == 0) && ((reinterpret_cast<uintptr_t>(w) & 3) == 0);
    if (pairs) {
        const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(w);
        for (int i = lane; i < K / 2; i += 32) {
            const float2 wf = __bfloat1622float2(w2[i]);
#pragma unroll
            for (int b = 0; b < BMAX; ++b)
                if (b < B) acc[b] = fmaf(wf.y, x[(int64_t)b * K + 2 * i + 1], fmaf(wf.x, x[(int64_t)b * K + 2 * i], acc[b]));
        }
    } else {
        for (int i = lane; i < K; i += 32) {
            const float wf = __bfloat162float(w[i]);
#pragma unroll
            for (int b = 0; b < BMAX; ++b)
                if (b < B) acc[b] = fmaf(wf, x[(int64_t)b * K + i], acc[b]);
        }
    }
#pragma unroll
    for (int b = 0; b < BMAX; ++b) {
        float v = acc[b];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0 && b < B) {
            v += bias ? bias[warp] : 0.f;
            y[(int64_t)b * N + warp] = v;
            if (yg) yg[(int64_t)b * N + warp] = gelu(v);
        }
    }
}

// y = x W^T + bias for x [B][K] (FP32), W [N][K] (BF16): GEMV below 5 rows, tiled GEMM above.
static void linear(int B, int N, int K, const float* x, const __nv_bfloat16* W, const float* bias, float* y, float* yg,
                   cudaStream_t s) {
    if (B <= 4) {
        k_gemv<4><<<(N * 32 + 255) / 256, 256, 0, s>>>(B, N, K, x, W, bias, y, yg);
        EQC_CHECK_LAUNCH();
        count_launch();
    } else {
        tile(OpRows<float, true>{x, K}, OpRows<__nv_bfloat16, true>{W, K}, EpLinear{{}, y, N, bias, yg}, B, N, K, s);
    }
}

// ---- convolution (kernel 5, stride 2, padding 2) ----------------------------------------
// z[b][co][t] = bias[co] + sum_{ci,k} W[co][ci][k] in[b][ci][2t+k-2] ; a = GELU(z)
__global__ void k_conv_fwd(const float* __restrict__ in, int Cin, int Tin, const __nv_bfloat16* __restrict__ W,
                           const float* __restrict__ bias, float* __restrict__ z, float* __restrict__ a, int Tout,
                           int B) {
    EQC_GRID_WAIT();
    const int64_t n = (int64_t)B * GN_C * Tout;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (int64_t)gridDim.x * blockDim.x) {
        const int t = (int)(idx % Tout);
        const int co = (int)((idx / Tout) % GN_C);
        const int b = (int)(idx / ((int64_t)Tout * GN_C));
        float acc = bias[co];
        const float* ib = in + (int64_t)b * Cin * Tin;
        const __nv_bfloat16* wc = W + (int64_t)co * Cin * GN_K;
        for (int ci = 0; ci < Cin; ++ci) {
#pragma unroll
            for (int k = 0; k < GN_K; ++k) {
                const int s = 2 * t + k - 2;
                if (s >= 0 && s < Tin) acc = fmaf(__bfloat162float(wc[ci * GN_K + k]), ib[(int64_t)ci * Tin + s], acc);
            }
        }
        z[idx] = acc;
        a[idx] = gelu(acc);
    }
}

// Mean squared error over B x nout: g = 2 (out - tgt) / (B nout); loss[b] = sum_j (out - tgt)^2
__global__ void __launch_bounds__(256) k_mse(const float* __restrict__ out, const float* __restrict__ tgt, int nout, int B,
                                             float* __restrict__ g, double* __restrict__ loss) {
    EQC_GRID_WAIT();
    const int b = blockIdx.x;
    const float sc = 2.f / ((float)B * (float)nout);
    double s = 0.0;
#pragma unroll 4
    for (int j = threadIdx.x; j < nout; j += blockDim.x) {
        const float e = out[(int64_t)b * nout + j] - tgt[(int64_t)b * nout + j];
        g[(int64_t)b * GN_LDOUT + j] = sc * e;
        const double d = f32_to_f64(e);
        s = fma(d, d, s);
    }
    if (threadIdx.x < GN_LDOUT - nout) g[(int64_t)b * GN_LDOUT + nout + threadIdx.x] = 0.f;   // the row's padding
    s = cta_sum(s);
    if (threadIdx.x == 0) loss[b] = s;
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int64_t n, float lr, float b1, float b2, float eps, float c1, float c2) {
    EQC_GRID_WAIT();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

__global__ void k_to_bf16(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, int64_t n) {
    EQC_GRID_WAIT();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = __float2bfloat16_rn(x[i]);
}

static inline int nblk(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 8 * 152); }

// ---- network set-up -------------------------------------------------------------------
void gn_reserve(GuessNet& g, int batch) {
    if (batch <= g.cap) return;
    g.cap = batch;
    g.x0.alloc((size_t)batch * 2 * g.T[0]);
    for (int l = 0; l < GN_LAYERS; ++l) {
        const size_t n = (size_t)batch * GN_C * g.T[l + 1];
        g.z[l].alloc(n);
        g.a[l].alloc(n);
        g.g_a[l].alloc(n);
    }
    g.zf1.alloc((size_t)batch * GN_NH);
    g.af1.alloc((size_t)batch * GN_NH);
    g.g_af1.alloc((size_t)batch * GN_NH);
    g.out.alloc((size_t)batch * g.nout);
    g.g_out.alloc((size_t)batch * GN_LDOUT);
    g.loss.alloc(batch);
}

void gn_init(Handle& h, uint64_t seed) {
    GuessNet& g = *h.net;
    g.Nf = h.F.Nf;
    g.T[0] = g.Nf;
    for (int l = 0; l < GN_LAYERS; ++l) g.T[l + 1] = (g.T[l] - 1) / 2 + 1;
    g.flat = GN_C * g.T[GN_LAYERS];
    int64_t o = 0;
    for (int l = 0; l < GN_LAYERS; ++l) {
        const int cin = l == 0 ? 2 : GN_C;
        g.off_cw[l] = o; o += (int64_t)GN_C * cin * GN_K;
        g.off_cb[l] = o; o += GN_C;
    }
    g.off_f1w = o; o += (int64_t)GN_NH * g.flat;
    g.off_f1b = o; o += GN_NH;
    g.off_f2w = o; o += (int64_t)g.nout * GN_NH;
    g.off_f2b = o; o += g.nout;
    g.nparam = o;
    // He-uniform weights (fan-in), zero biases, from a seeded stream
    std::vector<float> p(o, 0.f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int64_t off, int64_t n, int fan_in) {
        const float lim = std::sqrt(6.0f / (float)fan_in);
        std::uniform_real_distribution<float> U(-lim, lim);
        for (int64_t i = 0; i < n; ++i) p[off + i] = U(rng);
    };
    for (int l = 0; l < GN_LAYERS; ++l) {
        const int cin = l == 0 ? 2 : GN_C;
        fill(g.off_cw[l], (int64_t)GN_C * cin * GN_K, cin * GN_K);
    }
    fill(g.off_f1w, (int64_t)GN_NH * g.flat, g.flat);
    fill(g.off_f2w, (int64_t)g.nout * GN_NH, GN_NH);
    cudaStream_t s = h.stream;
    g.master.alloc(o);
    g.master.upload(p.data(), o, s);
    g.grad.alloc(o);
    g.m1.alloc(o);
    g.m2.alloc(o);
    g.wbf.alloc(o);
    g.w_part.alloc((size_t)GN_WSPLIT * GN_C * GT_N);
    g.b_part.alloc((size_t)GN_WSPLIT * GN_C);
    g.adam_t = 0;
    g.trained = false;
    gn_refresh_bf16(g, s);
    g.feat.alloc(2 * g.Nf);
    g.scale.alloc(1);
    gn_reserve(g, 1);
    EQC_CUDA(cudaStreamSynchronize(s));
}

void gn_refresh_bf16(GuessNet& g, cudaStream_t s) {
    k_to_bf16<<<nblk(g.nparam), 256, 0, s>>>(g.master.p, g.wbf.p, g.nparam);
    EQC_CHECK_LAUNCH();
    count_launch();
}

// ---- forward / backward ----------------------------------------------------------------
void gn_forward(GuessNet& g, const float* x0, int B, cudaStream_t s) {
    const float* in = x0;
    int cin = 2;
    for (int l = 0; l < GN_LAYERS; ++l) {
        const int64_t n = (int64_t)B * GN_C * g.T[l + 1];
        const __nv_bfloat16* W = g.wbf.p + g.off_cw[l];
        const float* bias = g.master.p + g.off_cb[l];
        if (B <= 4) {
            k_conv_fwd<<<nblk(n), 256, 0, s>>>(in, cin, g.T[l], W, bias, g.z[l].p, g.a[l].p, g.T[l + 1], B);
            EQC_CHECK_LAUNCH();
            count_launch();
        } else {
            tile(OpConvW{{}, W, cin * GN_K}, OpConvIn<false>{{}, in, cin, g.T[l], g.T[l + 1]},
                 EpConv{{}, g.z[l].p, g.a[l].p, bias, g.T[l + 1]}, GN_C, B * g.T[l + 1], cin * GN_K, s);
        }
        in = g.a[l].p;
        cin = GN_C;
    }
    // fc1: zf1 = a3 W1^T + b1, af1 = GELU(zf1) ; fc2: out = af1 W2^T + b2
    linear(B, GN_NH, g.flat, g.a[GN_LAYERS - 1].p, g.wbf.p + g.off_f1w, g.master.p + g.off_f1b, g.zf1.p, g.af1.p, s);
    linear(B, g.nout, GN_NH, g.af1.p, g.wbf.p + g.off_f2w, g.master.p + g.off_f2b, g.out.p, nullptr, s);
}

// Gradient of the mean squared error of g.out (after gn_forward on x0) against tgt.
void gn_backward(GuessNet& g, const float* x0, const float* tgt, int B, cudaStream_t s) {
    k_mse<<<B, 256, 0, s>>>(g.out.p, tgt, g.nout, B, g.g_out.p, g.loss.p);
    count_launch();
    // fc2: weight and bias, then g_z of fc1
    tile<false>(OpRows<float, false>{g.g_out.p, GN_LDOUT}, OpRows<float, false>{g.af1.p, GN_NH},
         EpWeight<false, false>{g.grad.p + g.off_f2w, g.grad.p + g.off_f2b, nullptr, g.nout, GN_NH, {}}, g.nout, GN_NH, B, s);
    tile(OpRows<float, true>{g.g_out.p, GN_LDOUT}, OpRows<__nv_bfloat16, false>{g.wbf.p + g.off_f2w, GN_NH},
         EpGeluGrad{{}, g.g_af1.p, g.zf1.p, GN_NH}, B, GN_NH, g.nout, s);
    // fc1: weight and bias, then g_z of the last convolution
    constexpr int last = GN_LAYERS - 1;
    tile<false>(OpRows<float, false>{g.g_af1.p, GN_NH}, OpRows<float, false>{g.a[last].p, g.flat},
         EpWeight<false, false>{g.grad.p + g.off_f1w, g.grad.p + g.off_f1b, nullptr, GN_NH, g.flat, {}}, GN_NH, g.flat, B, s);
    tile(OpRows<float, true>{g.g_af1.p, GN_NH}, OpRows<__nv_bfloat16, false>{g.wbf.p + g.off_f1w, g.flat},
         EpGeluGrad{{}, g.g_a[last].p, g.z[last].p, g.flat}, B, g.flat, GN_NH, s);
    // convolutions, last to first: weight and bias, then g_z of the layer below
    for (int l = last; l >= 0; --l) {
        const int cin = l == 0 ? 2 : GN_C, T = g.T[l + 1], N = cin * GN_K, K = B * T;
        const float* in = l == 0 ? x0 : g.a[l - 1].p;
        const int tiles = (N + GT_N - 1) / GT_N;
        const int chunk = std::max(256, (K / (GN_WSPLIT / tiles) + GT_K) / GT_K * GT_K);
        const dim3 grid(tiles, 1, (K + chunk - 1) / chunk);
        const EpWeight<true, true> ep{g.w_part.p, nullptr, g.b_part.p, GN_C, N, {}};
        k_tile<OpConvGz, OpConvIn<true>, EpWeight<true, true>, 1><<<grid, GT_THREADS, 0, s>>>(
            OpConvGz{{}, g.g_a[l].p, T}, OpConvIn<true>{{}, in, cin, g.T[l], T}, ep, GN_C, N, K, chunk);
        k_weight_sum<<<(GN_C * N + GN_C + 31) / 32, 256, 0, s>>>(g.w_part.p, g.b_part.p, grid.z, tiles, GN_C, N, g.grad.p + g.off_cw[l],
                                                           g.grad.p + g.off_cb[l]);
        EQC_CHECK_LAUNCH();
        count_launch(2);
        if (l > 0) {
            const __nv_bfloat16* W = g.wbf.p + g.off_cw[l];
            const int Ti = g.T[l], U0 = (Ti + 1) / 2, U1 = Ti / 2;
            tile(OpTapsW<3>{{}, W}, OpTapsGz<3>{{}, g.g_a[l].p, T, U0}, EpConvGrad{{}, g.g_a[l - 1].p, g.z[l - 1].p, Ti, U0, 0}, GN_C,
                 B * U0, GN_C * 3, s);
            tile(OpTapsW<2>{{}, W}, OpTapsGz<2>{{}, g.g_a[l].p, T, U1}, EpConvGrad{{}, g.g_a[l - 1].p, g.z[l - 1].p, Ti, U1, 1}, GN_C,
                 B * U1, GN_C * 2, s);
        }
    }
}

void gn_adam(GuessNet& g, double lr, cudaStream_t s) {
    g.adam_t += 1;
    const double b1 = 0.9, b2 = 0.999;
    const float c1 = (float)(1.0 - std::pow(b1, (double)g.adam_t)), c2 = (float)(1.0 - std::pow(b2, (double)g.adam_t));
    k_adam<<<nblk(g.nparam), 256, 0, s>>>(g.master.p, g.grad.p, g.m1.p, g.m2.p, g.nparam, (float)lr, (float)b1,
                                          (float)b2, 1e-8f, c1, c2);
    EQC_CHECK_LAUNCH();
    count_launch();
    gn_refresh_bf16(g, s);
}

// ---- coarse grid <-> GLL nodes ----------------------------------------------------------
// Position of lattice index i (4*nel+1 points) as a fraction of the axis.
__device__ __forceinline__ float node_frac(int i, int nel, const float* sk) {
    const int e = min(i >> 2, nel - 1);
    return ((float)e + sk[i - 4 * e]) / (float)nel;
}
// Lattice interval containing fraction f: lower index and weight of the upper one.
__device__ __forceinline__ void locate(float f, int nel, const float* sk, int& i0, float& w) {
    float u = f * (float)nel;
    int e = min(max((int)floorf(u), 0), nel - 1);
    const float loc = u - (float)e;
    int k = 0;
    while (k < 3 && loc > sk[k + 1]) ++k;
    i0 = 4 * e + k;
    w = (loc - sk[k]) / (sk[k + 1] - sk[k]);
    w = fminf(fmaxf(w, 0.f), 1.f);
}

struct GllFrac {
    float s[5];   // (1 + xi_k) / 2
};

// d[i] += s * P(out) and g32[i] = that increment, rows >= 1 (P bilinear from the coarse grid)
__global__ void k_guess_prolong(const float* __restrict__ out, const float* __restrict__ scale, double* __restrict__ d,
                                float* __restrict__ g32, Layout L, GllFrac f) {
    EQC_GRID_WAIT();
    const float sc = scale[0];
    const int64_t n = L.size();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int ix = (int)(i % L.ld), iy = (int)(i / L.ld);
        float v = 0.f;
        if (iy >= 1 && ix < L.nx && sc > 0.f) {
            const float gx = node_frac(ix, L.NelX, f.s) * (GN_GX - 1), gy = node_frac(iy, L.NelY, f.s) * (GN_GY - 1);
            const int i0 = min((int)gx, GN_GX - 2), j0 = min((int)gy, GN_GY - 2);
            const float wx = gx - (float)i0, wy = gy - (float)j0;
            const float* o = out + (int64_t)j0 * GN_GX + i0;
            v = sc * ((1.f - wy) * ((1.f - wx) * o[0] + wx * o[1]) + wy * ((1.f - wx) * o[GN_GX] + wx * o[GN_GX + 1]));
            d[i] += (double)v;
        }
        g32[i] = v;
    }
}

// Features of the first solve of a step: dF = d - dPre on the fault row, s = max |dF|,
// feat = [dF / s, log10(V / Vpl) / 4] with V = Vf0 (slip rate at the start of the step).
__global__ void __launch_bounds__(1024) k_guess_features(const double* __restrict__ d, const double* __restrict__ dPre,
                                                         const double* __restrict__ Vf0, int Nf, double Vpl,
                                                         float* __restrict__ feat, float* __restrict__ scale) {
    EQC_GRID_WAIT();
    __shared__ double sh[32];
    __shared__ double smax;
    double m = 0.0;
    for (int k = threadIdx.x; k < Nf; k += blockDim.x) m = fmax(m, fabs(d[k] - dPre[k]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) b = fmax(b, sh[q]);
        smax = b;
        scale[0] = (float)b;
    }
    __syncthreads();
    const double s = smax;
    for (int k = threadIdx.x; k < Nf; k += blockDim.x) {
        feat[k] = s > 0 ? (float)((d[k] - dPre[k]) / s) : 0.f;
        feat[Nf + k] = (float)(log10(fmax(Vf0[k], 1e-30) / Vpl) / 4.0);
    }
}

// Logged pair at slot *count: the features and the target (d - dPre) / s sampled at the
// coarse grid points (bilinear in the GLL lattice).
__global__ void k_guess_log(const float* __restrict__ feat, const float* __restrict__ scale, const double* __restrict__ d,
                            const double* __restrict__ dPre, Layout L, GllFrac f, int Nf, float* __restrict__ log_in,
                            float* __restrict__ log_tgt, const long long* __restrict__ count, long long cap) {
    EQC_GRID_WAIT();
    const long long c = *count;
    if (c >= cap) return;
    const float sc = scale[0];
    const int nin = 2 * Nf, nout = GN_GX * GN_GY;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nin + nout; j += gridDim.x * blockDim.x) {
        if (j < nin) {
            log_in[c * nin + j] = feat[j];
            continue;
        }
        const int q = j - nin, gi = q % GN_GX, gj = q / GN_GX;
        int i0, j0;
        float wx, wy;
        locate((float)gi / (GN_GX - 1), L.NelX, f.s, i0, wx);
        locate((float)gj / (GN_GY - 1), L.NelY, f.s, j0, wy);
        const int i1 = min(i0 + 1, L.nx - 1), j1 = min(j0 + 1, L.ny - 1);
        auto at = [&](int ix, int iy) {
            const int64_t p = (int64_t)iy * L.ld + ix;
            return (float)(d[p] - dPre[p]);
        };
        const float v = (1.f - wy) * ((1.f - wx) * at(i0, j0) + wx * at(i1, j0)) +
                        wy * ((1.f - wx) * at(i0, j1) + wx * at(i1, j1));
        log_tgt[c * nout + q] = sc > 0.f ? v / sc : 0.f;
    }
}
__global__ void k_guess_log_commit(long long* count, long long cap) {
    EQC_GRID_WAIT();
    if (*count < cap) *count += 1;
}

static GllFrac gll_frac() {
    static const double xg[5] = {-1.0, -0.65465367070797714, 0.0, 0.65465367070797714, 1.0};
    GllFrac f;
    for (int k = 0; k < 5; ++k) f.s[k] = (float)(0.5 * (1.0 + xg[k]));
    return f;
}

void gn_enqueue_features(Handle& h) {
    GuessNet& g = *h.net;
    k_guess_features<<<1, 1024, 0, h.stream>>>(h.d.p, h.dPre.p, h.F.Vf0.p, h.F.Nf, h.Vpl, g.feat.p, g.scale.p);
    EQC_CHECK_LAUNCH();
    count_launch();
}

void gn_enqueue_guess(Handle& h) {
    GuessNet& g = *h.net;
    gn_forward(g, g.feat.p, 1, h.stream);
    k_guess_prolong<<<nblk(h.L.size()), 256, 0, h.stream>>>(g.out.p, g.scale.p, h.d.p, h.g32.p, h.L, gll_frac());
    EQC_CHECK_LAUNCH();
    count_launch();
}

void gn_enqueue_log(Handle& h) {
    GuessNet& g = *h.net;
    const int n = 2 * g.Nf + GN_GX * GN_GY;
    k_guess_log<<<(n + 255) / 256, 256, 0, h.stream>>>(g.feat.p, g.scale.p, h.d.p, h.dPre.p, h.L, gll_frac(), g.Nf,
                                                       g.log_in.p, g.log_tgt.p, g.log_count.p, g.log_cap);
    k_guess_log_commit<<<1, 1, 0, h.stream>>>(g.log_count.p, g.log_cap);
    EQC_CHECK_LAUNCH();
    count_launch(2);
}

// ---- training ---------------------------------------------------------------------------
// x0[b] = pin[idx[b]], tgt[b] = ptgt[idx[b]]
__global__ void k_gather_batch(const float* __restrict__ pin, const float* __restrict__ ptgt, const int* __restrict__ idx,
                               int B, int nin, int nout, float* __restrict__ x0, float* __restrict__ tgt) {
    EQC_GRID_WAIT();
    const int64_t n = (int64_t)B * (nin + nout);
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(e / (nin + nout)), j = (int)(e % (nin + nout));
        const int64_t src = idx[b];
        if (j < nin) x0[(int64_t)b * nin + j] = pin[src * nin + j];
        else tgt[(int64_t)b * nout + (j - nin)] = ptgt[src * nout + (j - nin)];
    }
}
__global__ void k_sum_loss(const double* __restrict__ loss, int B, double* acc) {
    EQC_GRID_WAIT();
    double s = 0.0;
    for (int b = threadIdx.x; b < B; b += 32) s += loss[b];
    s = warp_sum(s);
    if (threadIdx.x == 0) *acc += s;
}

struct TrainBufs {
    DBuf<int> idx;
    DBuf<float> tgt;
    DBuf<double> acc;
};

// Trains on the n pairs resident in g.pin / g.ptgt; epoch_loss[e] = mean squared error per output.
static void gn_train(Handle& h, int64_t n, int epochs, double lr, int batch, uint64_t seed, double* epoch_loss) {
    GuessNet& g = *h.net;
    cudaStream_t s = h.stream;
    const int nin = 2 * g.Nf, nout = g.nout;
    batch = (int)std::max<int64_t>(1, std::min<int64_t>(batch, n));
    gn_reserve(g, batch);
    TrainBufs tb;
    tb.idx.alloc(n);
    tb.tgt.alloc((size_t)batch * nout);
    tb.acc.alloc(1);
    std::vector<int> perm(n);
    std::mt19937_64 rng(seed ^ 0x9e3779b97f4a7c15ull);
    for (int e = 0; e < epochs; ++e) {
        for (int64_t i = 0; i < n; ++i) perm[i] = (int)i;
        std::shuffle(perm.begin(), perm.end(), rng);
        tb.idx.upload(perm.data(), n, s);
        tb.acc.zero(s);
        for (int64_t b0 = 0; b0 + batch <= n; b0 += batch) {   // whole batches only
            k_gather_batch<<<nblk((int64_t)batch * (nin + nout)), 256, 0, s>>>(g.pin.p, g.ptgt.p, tb.idx.p + b0, batch,
                                                                             nin, nout, g.x0.p, tb.tgt.p);
            count_launch();
            gn_forward(g, g.x0.p, batch, s);
            gn_backward(g, g.x0.p, tb.tgt.p, batch, s);
            k_sum_loss<<<1, 32, 0, s>>>(g.loss.p, batch, tb.acc.p);
            count_launch();
            gn_adam(g, lr, s);
        }
        double acc = 0;
        tb.acc.download(&acc, 1, s);
        EQC_CUDA(cudaStreamSynchronize(s));
        const int64_t used = (n / batch) * batch;
        if (epoch_loss) epoch_loss[e] = used ? acc / ((double)used * nout) : 0.0;
    }
    EQC_CUDA(cudaStreamSynchronize(s));
    g.trained = true;
}

// Mean squared error per output over n pairs (batched forward); out (optional) gets the outputs.
static double gn_eval(Handle& h, int64_t n, float* out_host) {
    GuessNet& g = *h.net;
    cudaStream_t s = h.stream;
    const int nin = 2 * g.Nf, nout = g.nout;
    const int batch = (int)std::min<int64_t>(std::max<int64_t>(n, 1), 256);
    gn_reserve(g, batch);
    TrainBufs tb;
    tb.idx.alloc(batch);
    tb.tgt.alloc((size_t)batch * nout);
    tb.acc.alloc(1);
    tb.acc.zero(s);
    std::vector<int> ids(batch);
    for (int64_t b0 = 0; b0 < n; b0 += batch) {
        const int B = (int)std::min<int64_t>(batch, n - b0);
        for (int b = 0; b < B; ++b) ids[b] = (int)(b0 + b);
        tb.idx.upload(ids.data(), B, s);
        k_gather_batch<<<nblk((int64_t)B * (nin + nout)), 256, 0, s>>>(g.pin.p, g.ptgt.p, tb.idx.p, B, nin, nout,
                                                                       g.x0.p, tb.tgt.p);
        gn_forward(g, g.x0.p, B, s);
        k_mse<<<B, 256, 0, s>>>(g.out.p, tb.tgt.p, nout, B, g.g_out.p, g.loss.p);
        k_sum_loss<<<1, 32, 0, s>>>(g.loss.p, B, tb.acc.p);
        count_launch(3);
        if (out_host) g.out.download(out_host + b0 * nout, (size_t)B * nout, s);
        EQC_CUDA(cudaStreamSynchronize(s));
    }
    double acc = 0;
    tb.acc.download(&acc, 1, s);
    EQC_CUDA(cudaStreamSynchronize(s));
    return n ? acc / ((double)n * nout) : 0.0;
}

static void upload_pairs(Handle& h, const float* in, const float* tgt, int64_t n) {
    GuessNet& g = *h.net;
    const int nin = 2 * g.Nf, nout = g.nout;
    if ((int64_t)g.pin.n < n * nin) g.pin.alloc((size_t)n * nin);
    if ((int64_t)g.ptgt.n < n * nout) g.ptgt.alloc((size_t)n * nout);
    if (in) {
        g.pin.upload(in, (size_t)n * nin, h.stream);
        g.ptgt.upload(tgt, (size_t)n * nout, h.stream);
    } else {   // the pairs logged by this handle's time loop
        long long c = 0;
        g.log_count.download(&c, 1, h.stream);
        EQC_CUDA(cudaStreamSynchronize(h.stream));
        if (c < n) throw Error(EQC_E_ARG, "fewer logged pairs than requested");
        EQC_CUDA(cudaMemcpyAsync(g.pin.p, g.log_in.p, sizeof(float) * n * nin, cudaMemcpyDeviceToDevice, h.stream));
        EQC_CUDA(cudaMemcpyAsync(g.ptgt.p, g.log_tgt.p, sizeof(float) * n * nout, cudaMemcpyDeviceToDevice, h.stream));
    }
    g.npairs = n;
}

static GuessNet& net_of(Handle& h) {
    if (!h.net) {
        h.net = new GuessNet();
        gn_init(h, 1234);
    }
    return *h.net;
}

}  // namespace eqc

using namespace eqc;

template <class F>
static eqc_status guarded_net(eqc_handle* H, F&& f) {
    if (!H) return EQC_E_ARG;
    try {
        f(H->h);
        return EQC_OK;
    } catch (const Error& e) {
        H->h.err = e.what();
        return e.code;
    } catch (const std::exception& e) {
        H->h.err = e.what();
        return EQC_E_ARG;
    }
}

extern "C" {

eqc_status eqc_guess_shape(eqc_handle* H, int32_t* nin, int32_t* nout, int64_t* nparam) {
    return guarded_net(H, [&](Handle& h) {
        GuessNet& g = net_of(h);
        if (nin) *nin = 2 * g.Nf;
        if (nout) *nout = g.nout;
        if (nparam) *nparam = g.nparam;
    });
}

eqc_status eqc_guess_init(eqc_handle* H, uint64_t seed) {
    return guarded_net(H, [&](Handle& h) {
        net_of(h);
        gn_init(h, seed);
        destroy_graphs(h);
    });
}

eqc_status eqc_guess_get_params(eqc_handle* H, float* p) {
    if (!p) return EQC_E_ARG;
    return guarded_net(H, [&](Handle& h) {
        GuessNet& g = net_of(h);
        g.master.download(p, g.nparam, h.stream);
        EQC_CUDA(cudaStreamSynchronize(h.stream));
    });
}

eqc_status eqc_guess_set_params(eqc_handle* H, const float* p) {
    if (!p) return EQC_E_ARG;
    return guarded_net(H, [&](Handle& h) {
        GuessNet& g = net_of(h);
        g.master.upload(p, g.nparam, h.stream);
        gn_refresh_bf16(g, h.stream);
        g.m1.zero(h.stream);
        g.m2.zero(h.stream);
        g.adam_t = 0;
        g.trained = true;
        EQC_CUDA(cudaStreamSynchronize(h.stream));
        destroy_graphs(h);
    });
}

eqc_status eqc_guess_log(eqc_handle* H, int64_t capacity) {
    if (capacity < 0) return EQC_E_ARG;
    return guarded_net(H, [&](Handle& h) {
        GuessNet& g = net_of(h);
        g.log_cap = capacity;
        if (capacity > 0) {
            g.log_in.alloc((size_t)capacity * 2 * g.Nf);
            g.log_tgt.alloc((size_t)capacity * g.nout);
        } else {
            g.log_in.release();
            g.log_tgt.release();
        }
        g.log_count.alloc(1);
        destroy_graphs(h);
    });
}

eqc_status eqc_guess_pairs(eqc_handle* H, float* in, float* tgt, int64_t* n) {
    if (!n) return EQC_E_ARG;
    return guarded_net(H, [&](Handle& h) {
        GuessNet& g = net_of(h);
        long long c = 0;
        if (g.log_count.p) {
            g.log_count.download(&c, 1, h.stream);
            EQC_CUDA(cudaStreamSynchronize(h.stream));
        }
        *n = c;
        if (in && c) g.log_in.download(in, (size_t)c * 2 * g.Nf, h.stream);
        if (tgt && c) g.log_tgt.download(tgt, (size_t)c * g.nout, h.stream);
        EQC_CUDA(cudaStreamSynchronize(h.stream));
    });
}

eqc_status eqc_guess_train(eqc_handle* H, const float* in, const float* tgt, int64_t n, int32_t epochs, double lr,
                           int32_t batch, uint64_t seed, double* epoch_loss) {
    if (n < 1 || epochs < 1 || batch < 1 || !(lr > 0) || (in == nullptr) != (tgt == nullptr)) return EQC_E_ARG;
    return guarded_net(H, [&](Handle& h) {
        net_of(h);
        upload_pairs(h, in, tgt, n);
        gn_train(h, n, epochs, lr, batch, seed, epoch_loss);
        destroy_graphs(h);
    });
}

eqc_status eqc_guess_eval(eqc_handle* H, const float* in, const float* tgt, int64_t n, double* mse, float* out) {
    if (!in || !tgt || n < 1 || !mse) return EQC_E_ARG;
    return guarded_net(H, [&](Handle& h) {
        net_of(h);
        destroy_graphs(h);   // batch buffers may move
        upload_pairs(h, in, tgt, n);
        *mse = gn_eval(h, n, out);
    });
}

eqc_status eqc_guess_grad(eqc_handle* H, const float* in, const float* tgt, int64_t n, float* grad, double* loss) {
    if (!in || !tgt || n < 1 || !grad) return EQC_E_ARG;
    return guarded_net(H, [&](Handle& h) {
        GuessNet& g = net_of(h);
        destroy_graphs(h);   // batch buffers may move
        upload_pairs(h, in, tgt, n);
        gn_reserve(g, (int)n);
        EQC_CUDA(cudaMemcpyAsync(g.x0.p, g.pin.p, sizeof(float) * n * 2 * g.Nf, cudaMemcpyDeviceToDevice, h.stream));
        gn_forward(g, g.x0.p, (int)n, h.stream);
        gn_backward(g, g.x0.p, g.ptgt.p, (int)n, h.stream);
        g.grad.download(grad, g.nparam, h.stream);
        std::vector<double> l(n);
        g.loss.download(l.data(), n, h.stream);
        EQC_CUDA(cudaStreamSynchronize(h.stream));
        double t = 0;
        for (double v : l) t += v;
        if (loss) *loss = t / ((double)n * g.nout);
    });
}

}  // extern "C"
