// The CG scalars taken from a finished dot product (solver.cu, sem.cu), by one thread.
#pragma once
#include "model.h"

namespace eqc {

// pq: pq = t and alpha = rho / pq; else rho = t (the value before into rho_prev) and beta = rho / rho_prev.
__device__ __forceinline__ void cg_take_dot(CGState* S, double t, bool pq) {
    if (pq) {
        S->pq = t;
        S->alpha = S->rho / t;
        S->alpha32 = (float)S->alpha;
    } else {
        S->rho_prev = S->rho;
        S->rho = t;
        S->beta = t / S->rho_prev;
        S->beta32 = (float)S->beta;
    }
}

}  // namespace eqc
