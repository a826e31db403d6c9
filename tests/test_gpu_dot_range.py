"""The mixed solver's dot products of FP32 vectors are sums in FP64 over the threads: a residual far larger than the
right-hand side (a guess far off, a small slip), whose entries' squares are FP32 numbers and whose norm's square is
not, is solved like any other."""
import numpy as np
import pytest

from eqcycle_gb300 import EQC_MIXED, EQC_PC_AMG, EQC_PC_JACOBI, EQC_TOL_R0, Solver, preset, set_parameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", [EQC_PC_AMG, EQC_PC_JACOBI], ids=["amg", "jacobi"])
@pytest.mark.parametrize("variant", [0, 8])
def test_norm_beyond_fp32(eqclib, variant, precond):
    P = set_parameters(preset("homog48").replace(NelX=48, NelY=48))
    rng = np.random.default_rng(4)
    iFlt = P.iarray.iFlt - 1
    bulk = np.ones(P.int_.nglob, bool)
    bulk[iFlt] = False
    with Solver(P, precond=EQC_PC_JACOBI, apply_variant=2) as ref:
        d0, e = rng.uniform(-1, 1, P.int_.nglob), np.zeros(P.int_.nglob)
        e[iFlt] = rng.uniform(0.5, 1, len(iFlt))
        b = np.linalg.norm(ref.apply_K(e)[bulk])
        d0[iFlt] = 0.0
        r0 = ref.apply_K(d0)[bulk]
        F = e[iFlt] * (np.max(np.abs(r0)) / b / 3e18)      # |r| <= 3e18 |b|
        b = b * (F[0] / e[iFlt][0])
        assert (np.linalg.norm(r0) / b) ** 2 > 1e40
        with Solver(P, precision=EQC_MIXED, precond=precond, apply_variant=variant, tol_rule=EQC_TOL_R0) as s:
            d, it, rr = s.qs_solve(F, d0, tol=1e-6, maxit=4000)
        r = ref.apply_K(d)[bulk]
    assert it > 1 and np.linalg.norm(r) <= 1.01e-6 * np.linalg.norm(r0)
