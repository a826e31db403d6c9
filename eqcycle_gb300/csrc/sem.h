// The FP32 stiffness operator of the quasi-static solve on the spectral-element level (sem.cu), with the
// work before and after it in the same launch.
#pragma once
#include "model.h"
#include "mg_pt.cuh"

namespace eqc {

// What the operand u of t = K_II u is, formed as it is loaded.
enum SemLoad {
    SL_PLAIN,     // x
    SL_FIRST,     // Dinv b / theta: the first smoothing iterate from x = 0
    SL_PROLONG,   // x + P0 xc (stored to uout at the owned nodes)
    SL_DIR        // x + beta p: the CG direction from z = x and the direction before (stored to uout)
};
// What becomes of t at the owned nodes.
enum SemEpi {
    SE_STORE,     // out = t
    SE_CHEB,      // out = u + c1 (u - up) + c2 Dinv (b - t)
    SE_RESTRICT   // bc = P0^T (b - t), with the coarse level's first smoothing step
};
// The iterate before u of a Chebyshev step.
enum SemPrev { SP_NONE, SP_ZERO, SP_FIRST, SP_VEC };   // c1 = 0; 0; Dinv b / theta; the vector xp

struct SemOp {
    const float* x = nullptr;
    const float *b = nullptr, *dinv = nullptr, *xp = nullptr;
    float *out = nullptr, *uout = nullptr;
    float c1 = 0.f, c2 = 0.f, inv_theta = 0.f;
    const float* xc = nullptr;   // coarse vector of SL_PROLONG (vertex grid)
    float* bc = nullptr;         // coarse vector of SE_RESTRICT
    ChebFirst<float> first;
    GllW<float> w;
    // SL_DIR: the directions of even and odd iterations, by the iteration count in S
    float *p0 = nullptr, *p1 = nullptr;
    // sum over the owned nodes of out . b (dot = 1, into rho and beta) or of u . t (dot = 2, into pq and
    // alpha)
    int dot = 0;
    CGState* S = nullptr;
    double* part = nullptr;
    unsigned* count = nullptr;
};

// True when this handle's FP32 quasi-static operator runs here (apply_variant 0, at most one element in eight of
// several rigidities: classify_elements).
bool sem_usable(const Handle& h);
void sem_launch(Handle& h, SemLoad load, SemEpi epi, SemPrev prev, const SemOp& o);
double set_H_sem(const double* H, cudaStream_t s);   // returns Handle::sem_scale

}  // namespace eqc
