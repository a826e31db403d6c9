// The CG scalars taken from a finished dot product (solver.cu, sem.cu), by one thread.
#pragma once
#include "model.h"
#include "vec.cuh"
#include "reduce.cuh"

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

// End of a reliable update of the mixed solver (one thread): S->rr holds the exact residual's norm; decides
// whether the loop goes on.
__device__ __forceinline__ void cg_check_b(CGState* S, Ctrl* C, cudaGraphConditionalHandle hw, int use_cond) {
    if (S->done != 3) {
        if (S->need_update) {
            const double rs = sqrt(S->rr) * S->inv_sigma;
            // the true residual left the recurrence's (the FP32 recurrences drifted, e.g. from a
            // guess far from the solution): continue from the true residual with a fresh direction
            if (rs > 2.0 * S->res) {
                S->restart = 1;
                C->cg_restarts += 1;
            }
            S->res = rs;
            S->rmax = rs;
            S->need_update = 0;
            C->cg_updates += 1;
        }
        const double r = S->res;
        S->done = !isfinite(r) ? 3 : (r <= S->reltol ? 1 : (S->it >= S->maxit ? 2 : 0));
    }
    if (use_cond) cudaGraphSetConditional(hw, S->done == 0 ? 1u : 0u);
}

// One entry of the residual in FP32 and its share of the norm (integer scaling and rounding: FP64 is slow).
__device__ __forceinline__ float residual32(double r, int es, double sg, DotAcc<float>& acc) {
    const float f = f64_to_f32(pow2_scale(r, es, sg));
    acc.add(f, f);
    return f;
}
// The end of a launch that stored the residual (ResidualOut), by every thread of the grid.
__device__ __forceinline__ void residual_done(const ResidualOut& R, const DotAcc<float>& acc) {
    grid_sum(acc, R.part, R.count, [&](double t) {
        R.S->rr = t;
        R.S->dx_clear = 1;   // r64 is exact for x
        if (R.check) cg_check_b(R.S, R.C, R.hw, R.use_cond);
    });
}

}  // namespace eqc
