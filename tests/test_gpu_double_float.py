"""The double-float apply (k_apply_df), on meshes large enough for it, around the edges of its 31 x 6-element
tiles and with elements of one rigidity, of several and both, against the FP64 apply; and the mixed solver's
reliable updates with the residual written by the applies' launches, on the same edges.

A result is a sum of at most 4 x 2 lines of some 50 double-float operations of 2^-44 each at the size of
|K| |x|, which max |K x| on random x stands for: 8 sqrt(50) 2^-44 < 4e-12 at worst; the bound is a quarter of
that, 1e-12."""
import ctypes as C

import numpy as np
import pytest

from eqcycle_gb300 import EQC_MIXED, EQC_PC_AMG, EQC_PC_JACOBI, Solver, preset, set_parameters
from eqcycle_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _params(nelx, nely, material):
    rule = {"one": 0, "rectangle": 1, "trapezoid": 2, "per-node": 0}[material]
    cfg = preset("dz480").replace(NelX=nelx, NelY=nely, LY=24e3 * nely / nelx, damage=rule, ThickX=12e3, ThickY=9e3)
    P = set_parameters(cfg)
    if material == "per-node":   # every third element has a rigidity per node
        rng = np.random.default_rng(nelx * 100 + nely)
        P.mesh.W[:, :, ::3] *= rng.uniform(0.5, 2.0, P.mesh.W[:, :, ::3].shape)
    return P


def _apply(s, torch, x, dtype):
    y = torch.zeros_like(x)
    L.check(L.lib().eqc_apply_K_device(s.h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), dtype), s.h)
    L.check(L.lib().eqc_sync(s.h), s.h)
    return y.cpu().numpy()


@pytest.mark.parametrize("nelx,nely,material", [(154, 215, "one"), (155, 216, "rectangle"), (156, 217, "trapezoid"),
                                                (30, 1070, "per-node"), (1070, 31, "trapezoid")])
def test_double_float_apply_large(eqclib, nelx, nely, material):
    torch = pytest.importorskip("torch")
    with Solver(_params(nelx, nely, material), precond=EQC_PC_JACOBI) as s:
        nx, ny, ld = s.layout()
        x = torch.zeros(ny, ld, dtype=torch.float64)
        x[:, :nx] = torch.as_tensor(np.random.default_rng(3).uniform(-1, 1, (ny, nx)))
        x = x.cuda()
        y64, ydf = _apply(s, torch, x, 0), _apply(s, torch, x, 2)
    assert not np.any(ydf[:, nx:])               # row padding untouched
    assert np.max(np.abs(ydf - y64)) <= 1e-12 * np.max(np.abs(y64))


@pytest.mark.parametrize("nelx,nely,material", [(13, 15, "trapezoid"), (15, 17, "rectangle"), (155, 216, "rectangle"),
                                                (156, 217, "trapezoid")])
def test_residual_of_reliable_updates(eqclib, monkeypatch, nelx, nely, material):
    """A mixed solve is certified on the FP64 residual that its launches write: formed again by the plain-load
    FP64 apply it is the same up to that apply's rounding (the sum over 6e5 nodes of some ten roundings of 1e-16
    each at the size of K and F, over |b|: under 1e-12; 1e-11 is asked), whichever way the intermediate updates go."""
    P = _params(nelx, nely, material)
    F = np.random.default_rng(7).uniform(0.5e-2, 1e-2, P.int_.FltNglob)
    iFlt = P.iarray.iFlt - 1
    bulk = np.ones(P.int_.nglob, bool)
    bulk[iFlt] = False
    its = []
    for env in (None, "EQC_NO_DF_UPDATE"):
        if env:
            monkeypatch.setenv(env, "1")
        with Solver(P, precision=EQC_MIXED, precond=EQC_PC_AMG) as s, \
                Solver(P, precond=EQC_PC_JACOBI, apply_variant=2) as ref:
            d, it, rr = s.qs_solve(F, np.zeros(P.int_.nglob), tol=1e-9)
            e = np.zeros(P.int_.nglob)
            e[iFlt] = F
            r, b = ref.apply_K(d)[bulk], ref.apply_K(e)[bulk]
        assert np.array_equal(d[iFlt], F) and rr <= 1e-9
        assert abs(np.linalg.norm(r) / np.linalg.norm(b) - rr) <= 1e-11
        its.append(it)
    assert abs(its[0] - its[1]) <= 1
