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


@pytest.mark.parametrize("nelx,nely,material", [(155, 216, "one"), (181, 179, "trapezoid"), (1070, 31, "rectangle"),
                                                (37, 23, "per-node all")])
def test_double_float_apply_smooth(eqclib, nelx, nely, material):
    """A smooth field (K x small against |K| |x|, the cancellation that a residual has), on odd meshes that the
    double-float kernel serves: 1e-12 of the random case's scale, as the 240 x 480 mesh of test_apply_variants.py."""
    torch = pytest.importorskip("torch")
    P = _params(nelx, nely, material.replace(" all", ""))
    if material.endswith("all"):
        P.mesh.W[:] *= np.random.default_rng(5).uniform(0.5, 2.0, P.mesh.W.shape)
    with Solver(P, precond=EQC_PC_JACOBI) as s:
        nx, ny, ld = s.layout()
        x = torch.zeros(ny, ld, dtype=torch.float64)
        x[:, :nx] = torch.as_tensor(np.random.default_rng(3).uniform(-0.5, 0.5, (ny, nx)))
        scale = np.max(np.abs(_apply(s, torch, x.cuda(), 0)))
        ix = torch.arange(nx, dtype=torch.float64)[None, :]
        iy = torch.arange(ny, dtype=torch.float64)[:, None]
        x[:, :nx] = 0.3 + 1e-3 * ix + 2e-3 * iy + 1e-4 * torch.sin(0.05 * ix) * torch.cos(0.03 * iy)
        z64, zdf = _apply(s, torch, x.cuda(), 0), _apply(s, torch, x.cuda(), 2)
    assert not np.array_equal(z64, zdf)          # not the FP64 apply
    assert np.max(np.abs(zdf - z64)) <= 1e-12 * scale * float(x.abs().max()) / 0.5


@pytest.mark.parametrize("nelx,nely,material,variant", [(155, 216, "trapezoid", 0), (33, 29, "per-node all", 0),
                                                        (33, 29, "trapezoid", 3)])
def test_intermediate_updates_through_steps(eqclib, monkeypatch, nelx, nely, material, variant):
    """Quasi-static steps with the intermediate updates in double-float arithmetic and with each in FP64
    (EQC_NO_DF_UPDATE), on meshes where the two launch different kernels: iteration counts within one per solve,
    displacement and state to the solver tolerance's scale (the bounds of test_apply_variants.py)."""
    P = _params(nelx, nely, material.replace(" all", ""))
    if material.endswith("all"):
        P.mesh.W[:] *= np.random.default_rng(5).uniform(0.8, 1.25, P.mesh.W.shape)
    out = []
    for env in (None, "EQC_NO_DF_UPDATE"):
        if env:
            monkeypatch.setenv(env, "1")
        with Solver(P, precision=EQC_MIXED, precond=EQC_PC_AMG, cg_tol=1e-8, apply_variant=variant) as s:
            s.init(P.cfg.V_init)
            st = s.run(12)
            assert st["qs_steps"] == 12
            out.append((st["cg_iters"], st["qs_solves"], {k: s.state(k) for k in ("d", "psi", "tau")}))
    (it_df, solves, a), (it_64, _, b) = out
    assert abs(it_df - it_64) <= solves
    assert not np.array_equal(a["d"], b["d"])    # other roundings: not the same kernels
    for k in a:
        assert np.max(np.abs(a[k] - b[k])) <= 1e-6 * np.max(np.abs(b[k])), k
