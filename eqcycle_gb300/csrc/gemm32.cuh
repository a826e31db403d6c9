// C(m, n) = sum_k A(m, k) B(k, n) in FP32 on 64 x 64 tiles, for the learned guess's layers (learn.cu): a
// fully connected layer, a convolution and their gradients differ in where A, B and C lie, which the
// operand and epilogue types say.
//
// FP32 multiply-add issue bounds it.  128 threads with 8 x 4 outputs each: two of a thread's outputs
// are one 64-bit register, so that one fma.rn.f32x2 does both (each half rounded as fmaf rounds), 16
// of them to four shared-memory loads.  k in slices of 16 through two shared buffers; the next slice's
// operands are in registers while this one is multiplied.  Matrices whose rows start on 16-byte boundaries
// (OpRows) come four elements a load; a convolution's operands, gathered at stride 2, one by one.
//
// Where the tiles are few (M x N small, K long) the CTAs of a cluster share K and one tile, whose parts they
// add through distributed shared memory in rank order (S); where K is a batch's positions the parts go
// to memory (EpPart) and a second launch adds them in FP64.  Sums are in a fixed order either way.
#pragma once
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cstdint>
#include <type_traits>
#include "common.h"
#include "vec.cuh"

namespace eqc {

constexpr int GT_N = 64, GT_K = 16, GT_P = GT_N + 4, GT_THREADS = 128;

// The two parts of an operand's address: a pointer, from the index that neighbouring threads step through, and
// an offset, from the other; s is a coordinate whose sum over both has to lie in range.
template <class T>
struct TilePtr {
    const T* q;
    int s;
};
struct TileOff {
    int off, s;
};

// Operands: element (mn, k) for the product's 64 x 16 slice, 8 to a thread.  K_FAST: neighbouring threads load
// neighbouring k (else mn).  VEC: four neighbours to a load.
// Row-major matrix with 16-byte rows (FP32) or 8-byte ones (BF16): p[mn ld + k], or p[k ld + mn].  A load that
// starts below the bound may pass it by three, into the row's padding, which holds zeros.
template <class T, bool KF>
struct OpRows {
    static constexpr bool K_FAST = KF, VEC = true;
    const T* p;
    int ld;
    __device__ void get4(int mn, int k, uint32_t* v) const {
        const T* q = p + (KF ? (int64_t)mn * ld + k : (int64_t)k * ld + mn);
        if constexpr (sizeof(T) == 4) {
            const uint4 f = *reinterpret_cast<const uint4*>(q);
            v[0] = f.x;
            v[1] = f.y;
            v[2] = f.z;
            v[3] = f.w;
        } else {
            const uint2 f = *reinterpret_cast<const uint2*>(q);
            v[0] = f.x;
            v[1] = f.y;
        }
    }
    __device__ float value(const uint32_t (&v)[8], int i) const {
        if (sizeof(T) == 4) return __uint_as_float(v[i]);
        const uint32_t w = v[i / 4 * 4 + i % 4 / 2];
        return __uint_as_float(i % 2 ? w & 0xffff0000u : w << 16);
    }
};

// Sums over k of A's rows beside the product (a bias's gradient from a weight's): in FP64, in
// the threads that load A; done calls f(m, sum).  For the two ways in which a weight gradient's A is loaded.
template <bool KF>
struct RowSum {
    static constexpr int R = KF ? 8 : 4;
    double s[R] = {};
    __device__ __forceinline__ void add(const float (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i % R] += f32_to_f64(v[i]);
    }
    template <class F>
    __device__ __forceinline__ void done(int m0, int M, F f) const {
        const int tid = threadIdx.x;
        if constexpr (KF) {   // one by one: rows (tid >> 4) + 8 i, of 16 threads
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                double d = s[i];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) d += __shfl_down_sync(0xffffffffu, d, o, 16);
                const int m = m0 + (tid >> 4) + 8 * i;
                if ((tid & 15) == 0 && m < M) f(m, d);
            }
        } else {              // four a load: rows 4 (tid & 15) + i, of 8 threads
            __shared__ double part[8][GT_N];
#pragma unroll
            for (int i = 0; i < 4; ++i) part[tid >> 4][4 * (tid & 15) + i] = s[i];
            __syncthreads();
            if (tid < GT_N && m0 + tid < M) {
                double d = 0.0;
                for (int q = 0; q < 8; ++q) d += part[q][tid];
                f(m0 + tid, d);
            }
        }
    }
};

template <class OA, class OB, class EP, int S>   // S: CTAs of a cluster along z that share a tile's K
__global__ void __launch_bounds__(GT_THREADS) k_tile(OA A, OB B, EP E, int M, int N, int K, int kchunk) {
    EQC_GRID_WAIT();
    __shared__ __align__(16) float sm[4 * GT_K * GT_P];
    const int tid = threadIdx.x, m0 = blockIdx.y * GT_N, n0 = blockIdx.x * GT_N;
    const int kb = blockIdx.z * kchunk, ke = min(K, kb + kchunk);
    // A slice's operands as loaded, and which of them count.  The loads have no condition (addresses are
    // clamped) and nothing reads them before the slice in hand is multiplied: under a branch each they came one
    // after the other.
    uint32_t va[8], vb[8];
    unsigned ina = 0, inb = 0;
    auto fetch = [&](auto& O, int o0, int lim, int k0, uint32_t (&v)[8], unsigned& in) {
        using Op = std::remove_cv_t<std::remove_reference_t<decltype(O)>>;
        in = 0;
        if constexpr (Op::VEC) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int mn = o0 + (Op::K_FAST ? (tid >> 2) + 32 * i : 4 * (tid & 15));
                const int k = k0 + (Op::K_FAST ? 4 * (tid & 3) : (tid >> 4) + 8 * i);
                const bool ok = mn < lim && k < ke;
                in |= ok ? 15u << (4 * i) : 0u;
                O.get4(ok ? mn : 0, ok ? k : 0, v + 4 * i);
            }
        } else {
            const int f = Op::K_FAST ? k0 + (tid & 15) : o0 + (tid & 63), fl = Op::K_FAST ? ke : lim;
            const auto q = O.ptr(min(f, fl - 1));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int g = Op::K_FAST ? o0 + (tid >> 4) + 8 * i : k0 + (tid >> 6) + 2 * i, gl = Op::K_FAST ? lim : ke;
                bool ok = true;
                v[i] = O.get(q, O.off(min(g, gl - 1)), ok);
                in |= ok && f < fl && g < gl ? 1u << i : 0u;
            }
        }
    };
    auto store = [&](auto& O, const float (&v)[8], auto put) {   // put(k, mn, value)
        using Op = std::remove_cv_t<std::remove_reference_t<decltype(O)>>;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (Op::VEC && Op::K_FAST) put(4 * (tid & 3) + (i & 3), (tid >> 2) + 32 * (i >> 2), v[i]);
            else if (Op::VEC) put((tid >> 4) + 8 * (i >> 2), 4 * (tid & 15) + (i & 3), v[i]);
            else if (Op::K_FAST) put(tid & 15, (tid >> 4) + 8 * i, v[i]);
            else put((tid >> 6) + 2 * i, tid & 63, v[i]);
        }
    };
    const int tx = tid & 15, ty = tid >> 4;   // outputs m = 8 ty + 0..7, n = 2 tx + {0, 1, 32, 33}
    unsigned long long acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    const int slices = (max(ke - kb, 0) + GT_K - 1) / GT_K;
    if (slices) {
        fetch(A, m0, M, kb, va, ina);
        fetch(B, n0, N, kb, vb, inb);
    }
    for (int t = 0; t < slices; ++t) {
        float* as = sm + (t & 1) * 2 * GT_K * GT_P;
        float* bs = as + GT_K * GT_P;
        float fa[8], fb[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            fa[i] = ina >> i & 1 ? A.value(va, i) : 0.f;
            fb[i] = inb >> i & 1 ? B.value(vb, i) : 0.f;
        }
        E.sum(fa, t);
        store(A, fa, [&](int k, int m, float v) { as[k * GT_P + m] = v; });
        store(B, fb, [&](int k, int n, float v) { bs[k * GT_P + n] = v; });
        __syncthreads();   // the other buffer's readers are past it too: they stored to this one after reading
        if (t + 1 < slices) {
            fetch(A, m0, M, kb + (t + 1) * GT_K, va, ina);
            fetch(B, n0, N, kb + (t + 1) * GT_K, vb, inb);
        }
#pragma unroll
        for (int k = 0; k < GT_K; ++k) {
            const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(as + k * GT_P + 8 * ty);
            const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(as + k * GT_P + 8 * ty + 4);
            const float2 b0 = *reinterpret_cast<const float2*>(bs + k * GT_P + 2 * tx);
            const float2 b1 = *reinterpret_cast<const float2*>(bs + k * GT_P + 2 * tx + 32);
            const unsigned long long a[4] = {a0.x, a0.y, a1.x, a1.y};
            const float b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                unsigned long long bb;
                asm("mov.b64 %0, {%1, %1};" : "=l"(bb) : "f"(b[j]));
#pragma unroll
                for (int i = 0; i < 4; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a[i]), "l"(bb));
            }
        }
    }
    E.sum_done(m0, n0, M);
    float c[8][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) asm("mov.b64 {%0, %1}, %2;" : "=f"(c[2 * i][j]), "=f"(c[2 * i + 1][j]) : "l"(acc[i][j]));
    if constexpr (S == 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + 2 * tx + (j & 1) + 32 * (j >> 1);
            if (n >= N) continue;
            const int64_t np = E.npos(n);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int m = m0 + 8 * ty + i;
                if (m < M) E.put(m, n, np, c[i][j]);
            }
        }
    } else {
        namespace cg = cooperative_groups;
        auto cl = cg::this_cluster();
        static_assert(sizeof(sm) >= sizeof(float) * GT_N * GT_N && S <= 8, "a tile's part fits");
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            *reinterpret_cast<float2*>(sm + (8 * ty + i) * GT_N + 2 * tx) = make_float2(c[i][0], c[i][1]);
            *reinterpret_cast<float2*>(sm + (8 * ty + i) * GT_N + 2 * tx + 32) = make_float2(c[i][2], c[i][3]);
        }
        cl.sync();
        // this CTA's 64 / S rows of every part: the eight loads of a thread are in flight together
        float4 v[8 / S][S];
#pragma unroll
        for (int u = 0; u < 8 / S; ++u)
#pragma unroll
            for (int q = 0; q < S; ++q)
                v[u][q] = *reinterpret_cast<const float4*>(
                    cl.map_shared_rank(sm, q) + (8 / S * (int)cl.block_rank() + u) * 512 + 4 * tid);
        cl.sync();   // no CTA leaves while its part is being read
#pragma unroll
        for (int u = 0; u < 8 / S; ++u) {
            float4 t = v[u][0];
#pragma unroll
            for (int q = 1; q < S; ++q) {
                t.x += v[u][q].x;
                t.y += v[u][q].y;
                t.z += v[u][q].z;
                t.w += v[u][q].w;
            }
            const int f = (8 / S * (int)cl.block_rank() + u) * 512 + 4 * tid, m = m0 + f / GT_N, n = n0 + f % GT_N;
            const float w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (m < M && n + k < N) E.put(m, n + k, E.npos(n + k), w[k]);
        }
    }
}

}  // namespace eqc
