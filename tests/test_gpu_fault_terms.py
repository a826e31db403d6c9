"""The pair of exponentials of the slip-rate law (fault.cuh's exp_pair) on both sides of its switch at 20
and of its overflow limit: Vf = 2 Vo e^h sinh(fa) with fa = tau / (a sigma) from 1 to 900 against numpy
on the same state.  Both sides round h + fa and h - fa alike and their exponentials err by at most two
units in the last place each: 8 eps relative, infinities alike."""
import numpy as np
import pytest

from eqcycle_gb300 import EQC_PC_JACOBI, Solver, preset, set_parameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(1.0, 19.9), (19.9, 20.1), (20.1, 80.0), (600.0, 900.0)])
def test_slip_rate_over_the_switch(eqclib, lo, hi):
    P = set_parameters(preset("homog48"))
    f, n = P.farray, P.int_.FltNglob
    rng = np.random.default_rng(5)
    psi, Vf = rng.uniform(5.0, 25.0, n), 10 ** rng.uniform(-11, -1, n)
    tau1 = rng.uniform(lo, hi, n) * (f.Seff * f.cca) - f.tauo
    with Solver(P, precond=EQC_PC_JACOBI) as s:
        psi1, V = s.slrFunc(psi, np.zeros(n), Vf, np.zeros(n), tau1, 1e3)
    fa, h = (tau1 + f.tauo) / (f.Seff * f.cca), -(f.fo + f.ccb * psi1) / f.cca
    with np.errstate(over="ignore"):
        ref = f.Vo * (np.exp(h + fa) - np.exp(h - fa))
    on = psi1 != 0                                  # the friction nodes
    big = np.isinf(ref)
    assert on.sum() > n // 2
    assert np.array_equal(np.isinf(V[on]), big[on])
    ok = on & ~big
    assert np.all(np.abs(V[ok] - ref[ok]) <= 8 * np.finfo(float).eps * np.abs(ref[ok]))
