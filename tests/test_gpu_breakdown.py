"""A quasi-static solve that breaks down (EQC_E_NAN) leaves nothing behind: the next solve on the same handle gives
what a fresh handle gives, bit for bit.

The breakdown is made by the model: damage scales the rigidity of a few elements off the fault by 1e200, which
FP32 holds as infinity, so that the mixed method's first step length is not a number (the plain method stays in
range: it may solve or reach its iteration limit); damage by 1e-200 takes it back (the rigidities to a rounding, so the
fresh handle goes the same way)."""
import numpy as np
import pytest

from eqcycle_gb300 import EQC_FP64, EQC_MIXED, EQC_PC_AMG, EQC_PC_JACOBI, Solver, preset, set_parameters
from eqcycle_gb300._lib import EqcError

pytestmark = pytest.mark.gpu

E_CG, E_NAN = 4, 5
PRECISIONS = [pytest.param(EQC_FP64, id="fp64"), pytest.param(EQC_MIXED, id="mixed")]


def _params():
    """NelX even: the row padding holds seven nodes."""
    return set_parameters(preset("homog48").replace(NelX=12, NelY=16, LX=6e3, LY=8e3, creep_depth=6e3))


def _scale(s, els, factor):
    s.set_damage(els, factor)
    s.damage_evolve()


@pytest.mark.parametrize("precond", [EQC_PC_AMG, EQC_PC_JACOBI], ids=["amg", "jacobi"])
@pytest.mark.parametrize("variant", [0, 3, 8])
@pytest.mark.parametrize("precision", PRECISIONS)
def test_solves_after_a_breakdown(eqclib, precision, variant, precond):
    P = _params()
    els = np.arange(100, 104) + 1
    F = np.random.default_rng(2).uniform(0.5e-2, 1e-2, P.int_.FltNglob)
    d0 = np.zeros(P.int_.nglob)
    got = []
    for broken in (True, False):
        with Solver(P, precision=precision, precond=precond, apply_variant=variant) as s:
            _scale(s, els, 1e200)
            if broken:
                status = 0
                try:
                    s.qs_solve(F, d0, tol=1e-8, maxit=400)
                except EqcError as e:
                    status = e.status
                assert status == E_NAN if precision == EQC_MIXED else status in (0, E_CG)
            _scale(s, els, 1e-200)
            got.append(s.qs_solve(F, d0, tol=1e-8))
    assert got[0][1] == got[1][1] and got[0][2] == got[1][2] <= 1e-8
    assert np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("precision", PRECISIONS)
def test_solves_after_an_unreachable_tolerance(eqclib, precision):
    """No slip and a guess off the solution: |b| = 0, so the solve goes on until its numbers underflow.  It may end
    in a breakdown or in the zero solution; the handle keeps solving."""
    P = _params()
    rng = np.random.default_rng(3)
    d0 = rng.uniform(-1e-3, 1e-3, P.int_.nglob)
    F = rng.uniform(0.5e-2, 1e-2, P.int_.FltNglob)
    with Solver(P, precision=precision, precond=EQC_PC_AMG) as s:
        try:
            s.qs_solve(np.zeros_like(F), d0, tol=1e-8, maxit=2000)
        except EqcError:
            pass
        d, it, rr = s.qs_solve(F, np.zeros_like(d0), tol=1e-8)
    with Solver(P, precision=precision, precond=EQC_PC_AMG) as s:
        e, jt, qq = s.qs_solve(F, np.zeros_like(d0), tol=1e-8)
    assert it == jt and rr == qq <= 1e-8 and np.array_equal(d, e)
