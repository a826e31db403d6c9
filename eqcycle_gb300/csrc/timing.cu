// Kernel timing with CUDA events on the handle's stream (used by bench.py for the
// roofline figure of the stiffness apply).
#include "model.h"

namespace eqc {

// L2 flush by reading a buffer larger than L2: afterwards L2 holds clean lines only, so the
// timed kernel pays no write-back of someone else's dirty data (a read-modify-write flush
// would leave L2 full of dirty lines and inflate the next kernel's DRAM traffic).
__global__ void k_flush(const float4* __restrict__ buf, int64_t n4, float* sink) {
    EQC_GRID_WAIT();
    float s = 0.f;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 v = buf[i];
        s += v.x + v.y + v.z + v.w;
    }
    if (s == 1.2345f) *sink = s;   // keeps the loads; the buffer holds zeros, so never taken
}

}  // namespace eqc

using namespace eqc;

extern "C" eqc_status eqc_time_apply(eqc_handle* H, int32_t dtype, int32_t nrep, int32_t flush_l2, double* ms) {
    if (!H || !ms || nrep < 1 || dtype < 0 || dtype > 2) return EQC_E_ARG;
    Handle& h = H->h;
    try {
        cudaStream_t s = h.stream;
        const int64_t N = h.L.size();
        const size_t es = dtype == 1 ? sizeof(float) : sizeof(double);
        void *x = nullptr, *y = nullptr;
        float* fl = nullptr;
        const int64_t nfl = (int64_t)(512ull << 20) / 4;  // 512 MB > L2
        EQC_CUDA(cudaMalloc(&x, N * es));
        EQC_CUDA(cudaMalloc(&y, N * es));
        if (flush_l2) EQC_CUDA(cudaMalloc(&fl, nfl * 4));
        EQC_CUDA(cudaMemsetAsync(x, 0, N * es, s));
        if (fl) EQC_CUDA(cudaMemsetAsync(fl, 0, nfl * 4, s));
        cudaEvent_t e0, e1;
        EQC_CUDA(cudaEventCreate(&e0));
        EQC_CUDA(cudaEventCreate(&e1));
        double tot = 0;
        for (int r = -2; r < nrep; ++r) {
            if (fl) {
                k_flush<<<8 * 152, 256, 0, s>>>(reinterpret_cast<const float4*>(fl), nfl / 4, fl);
                count_launch();
            }
            EQC_CUDA(cudaEventRecord(e0, s));
            if (dtype == 0) apply_K<double>((const double*)x, (double*)y, args64(h), 1.0, 0, s);
            else if (dtype == 1) apply_K<float>((const float*)x, (float*)y, args32(h), 1.0f, 0, s);
            else if (!apply_K_df(h, (const double*)x, (double*)y, 1.0, 0, s))
                throw Error(EQC_E_STATE, "double-float apply unavailable");
            EQC_CUDA(cudaEventRecord(e1, s));
            EQC_CUDA(cudaEventSynchronize(e1));
            float t = 0;
            EQC_CUDA(cudaEventElapsedTime(&t, e0, e1));
            if (r >= 0) tot += t;
        }
        *ms = tot / nrep;
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        cudaFree(x);
        cudaFree(y);
        if (fl) cudaFree(fl);
        return EQC_OK;
    } catch (const Error& e) {
        h.err = e.what();
        return e.code;
    }
}

// Streamed timing: `ncopies` replicas of the apply's whole working set (x, y, W and its padded
// copy) rotate through `nrep` back-to-back launches, so every launch reads its data from HBM
// once the replicas together exceed L2, and launch latency overlaps the previous launch as it
// does inside a solve; *ms gets the mean launch duration over the batch (CUDA events around it).
extern "C" eqc_status eqc_time_apply_stream(eqc_handle* H, int32_t dtype, int32_t nrep, int32_t ncopies,
                                            double* ms) {
    if (!H || !ms || nrep < 1 || ncopies < 1 || (dtype != 0 && dtype != 1)) return EQC_E_ARG;
    Handle& h = H->h;
    struct Replica {
        void *x = nullptr, *y = nullptr, *W = nullptr, *Wp = nullptr;
        float* W32p = nullptr;
        double* W64p = nullptr;
        TmaCache tma;
    };
    std::vector<Replica> R((size_t)ncopies);
    auto release = [&] {
        for (Replica& r : R) {
            for (void* p : {r.x, r.y, r.W, (void*)r.W32p, (void*)r.W64p}) if (p) cudaFree(p);
            r = Replica();
        }
    };
    try {
        cudaStream_t s = h.stream;
        const int64_t N = h.L.size(), Nel = (int64_t)h.L.NelX * h.L.NelY;
        const size_t es = dtype == 0 ? sizeof(double) : sizeof(float);
        for (Replica& r : R) {
            EQC_CUDA(cudaMalloc(&r.x, N * es));
            EQC_CUDA(cudaMalloc(&r.y, N * es));
            EQC_CUDA(cudaMalloc(&r.W, (size_t)25 * Nel * es));
            EQC_CUDA(cudaMalloc(&r.W32p, sizeof(float) * WPad<float>::v * Nel));
            EQC_CUDA(cudaMalloc(&r.W64p, sizeof(double) * WPad<double>::v * Nel));
            EQC_CUDA(cudaMemsetAsync(r.x, 0, N * es, s));
            EQC_CUDA(cudaMemcpyAsync(r.W, dtype == 0 ? (const void*)h.W64.p : (const void*)h.W32.p,
                                     (size_t)25 * Nel * es, cudaMemcpyDeviceToDevice, s));
            EQC_CUDA(cudaMemcpyAsync(r.W32p, h.W32p.p, sizeof(float) * WPad<float>::v * Nel, cudaMemcpyDeviceToDevice, s));
            EQC_CUDA(cudaMemcpyAsync(r.W64p, h.W64p.p, sizeof(double) * WPad<double>::v * Nel, cudaMemcpyDeviceToDevice,
                                     s));
            tma_init_for(r.tma, h.L, r.W32p, r.W64p, h.mu64.p);
        }
        EQC_CUDA(cudaStreamSynchronize(s));
        auto launch = [&](Replica& r) {
            if (dtype == 0) {
                ApplyArgs<double> A = args64(h);
                A.W = (const double*)r.W;
                A.Wp = r.W64p;
                A.tma = h.tma.ok ? &r.tma : nullptr;
                apply_K<double>((const double*)r.x, (double*)r.y, A, 1.0, 0, s);
            } else {
                ApplyArgs<float> A = args32(h);
                A.W = (const float*)r.W;
                A.Wp = r.W32p;
                A.tma = h.tma.ok ? &r.tma : nullptr;
                apply_K<float>((const float*)r.x, (float*)r.y, A, 1.0f, 0, s);
            }
        };
        for (int k = 0; k < 2 * ncopies; ++k) launch(R[(size_t)k % ncopies]);   // warm-up, maps encoded
        // the batch runs as the solver's step graphs run their kernels: captured in a graph whose
        // kernel-to-kernel edges are programmatic (each launch's CTAs start as its predecessor's
        // finish; what a kernel does before its grid-dependency wait overlaps the predecessor)
        cudaGraph_t g = nullptr;
        cudaGraphExec_t ge = nullptr;
        EQC_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        for (int k = 0; k < nrep; ++k) launch(R[(size_t)k % ncopies]);
        EQC_CUDA(cudaStreamEndCapture(s, &g));
        make_programmatic(g);
        EQC_CUDA(cudaGraphInstantiate(&ge, g, 0));
        EQC_CUDA(cudaGraphLaunch(ge, s));   // warm-up of the graph
        cudaEvent_t e0, e1;
        EQC_CUDA(cudaEventCreate(&e0));
        EQC_CUDA(cudaEventCreate(&e1));
        EQC_CUDA(cudaEventRecord(e0, s));
        EQC_CUDA(cudaGraphLaunch(ge, s));
        EQC_CUDA(cudaEventRecord(e1, s));
        EQC_CUDA(cudaEventSynchronize(e1));
        float t = 0;
        EQC_CUDA(cudaEventElapsedTime(&t, e0, e1));
        *ms = (double)t / nrep;
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        cudaGraphExecDestroy(ge);
        cudaGraphDestroy(g);
        release();
        return EQC_OK;
    } catch (const Error& e) {
        release();
        h.err = e.what();
        return e.code;
    }
}

