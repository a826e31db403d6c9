"""The FP32 spectral-element operator of the quasi-static solve (sem.cu) at the edges of its strips of 31
element columns and of its row walks, with elements of one rigidity and of several, and for every
number of smoothing steps.

The V-cycle with its vector work in the operator's launches and the one of separate kernels
(EQC_NO_FUSE) share their arithmetic point by point and differ in the order in which two dot
products per iteration are summed, as pairs of about 44 bits whose total is rounded to FP32: the CG
iterations are equal and the states agree bit for bit unless such a total lies within 2^-20 of a
rounding boundary; they are held to 1e-9.  Against the TMA-fed apply (variant 8), which takes both
contractions of every line, both solvers stop at the same residual (1e-10): displacement, state and
stress agree to 1e-6 of the largest entry (v, a difference of displacements over dt, carries the
stopping error divided by the step's displacement: 2e-4 on the smallest mesh, by either apply)."""
import numpy as np
import pytest

from eqcycle_gb300 import EQC_GUESS_EXTRAPOLATE, EQC_MIXED, Solver, preset, set_parameters

pytestmark = pytest.mark.gpu


def _steps(P, monkeypatch, no_fuse, **kw):
    if no_fuse:
        monkeypatch.setenv("EQC_NO_FUSE", "1")
    else:
        monkeypatch.delenv("EQC_NO_FUSE", raising=False)
    with Solver(P, precision=EQC_MIXED, guess=EQC_GUESS_EXTRAPOLATE, cg_tol=1e-10, **kw) as s:
        s.init(2 * P.cfg.Vpl)
        s.set_scalar("dt", 1e6)
        st = s.run(4)
        return st["cg_iters"], {k: s.state(k) for k in ("d", "v", "psi", "tau")}


@pytest.mark.parametrize("several", [False, True], ids=["one-rigidity", "several"])
@pytest.mark.parametrize("nelx,nely,deg,degc", [(4, 4, 1, 1), (5, 9, 2, 2), (29, 33, 3, 1), (30, 31, 4, 3), (31, 60, 4, 1),
                                                (62, 40, 5, 2), (93, 130, 2, 3), (200, 410, 3, 1)])
def test_fused_cycle_matches_separate_kernels(eqclib, monkeypatch, nelx, nely, deg, degc, several):
    P = set_parameters(preset("dz480").replace(NelX=nelx, NelY=nely, LY=24e3 * nely / nelx, damage=0))
    if several:   # one element in 29 with a rigidity per node: both forms of a line, mixed in a strip
        W = P.mesh.W[:, :, ::29]
        W *= np.random.default_rng(1).uniform(0.7, 1.4, W.shape)
    kw = dict(mg_degree=deg, mg_degree_coarse=degc)
    it0, a = _steps(P, monkeypatch, False, **kw)
    it1, b = _steps(P, monkeypatch, True, **kw)
    it2, c = _steps(P, monkeypatch, False, apply_variant=8, **kw)
    assert it0 == it1 > 0
    assert abs(it0 - it2) <= 8       # one iteration per solve
    for k in a:
        top = np.max(np.abs(b[k]))
        assert np.max(np.abs(a[k] - b[k])) <= 1e-9 * top, k
        assert k == "v" or np.max(np.abs(a[k] - c[k])) <= 1e-6 * top, k
