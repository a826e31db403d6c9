"""Models most of whose elements have several rigidities (W given per node, as eqc_create accepts it): the applies
that take both contractions of every line serve them, on meshes around the edges of the tiles, and the mixed solver's
residual is what the plain-load FP64 apply gives.

The double-float apply's bound of 1e-12 of max |K x| is test_gpu_double_float.py's (8 sqrt(50) 2^-44 < 4e-12 at
worst, a quarter of it asked)."""
import ctypes as C

import numpy as np
import pytest

from eqcycle_gb300 import EQC_MIXED, EQC_PC_AMG, EQC_PC_JACOBI, Solver, preset, set_parameters
from eqcycle_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _params(nelx, nely, share=1.0):
    cfg = preset("dz480").replace(NelX=nelx, NelY=nely, LY=24e3 * nely / nelx, damage=0)
    P = set_parameters(cfg)
    rng = np.random.default_rng(nelx * 100 + nely)
    el = rng.permutation(nelx * nely)[:int(np.ceil(share * nelx * nely))]
    P.mesh.W[:, :, el] *= rng.uniform(0.5, 2.0, (5, 5, len(el)))
    return P


def _apply(s, torch, dtype):
    nx, ny, ld = s.layout()
    x = torch.zeros(ny, ld, dtype=torch.float64)
    x[:, :nx] = torch.as_tensor(np.random.default_rng(3).uniform(-1, 1, (ny, nx)))
    x, y = x.cuda(), torch.zeros(ny, ld, dtype=torch.float64, device="cuda")
    L.check(L.lib().eqc_apply_K_device(s.h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), dtype), s.h)
    L.check(L.lib().eqc_sync(s.h), s.h)
    assert not bool(y[:, nx:].any())             # row padding untouched
    return y.cpu().numpy()


@pytest.mark.parametrize("share", [0.5, 1.0])
@pytest.mark.parametrize("nelx,nely", [(1, 1), (6, 8), (7, 9), (8, 7), (15, 17), (63, 65)])
def test_fp64_apply_takes_the_two_contraction_kernel(eqclib, nelx, nely, share):
    """Scattered over half of the elements they are in every tile: variant 0 gives the bits of variant 3, the
    pipelined kernel with both contractions."""
    torch = pytest.importorskip("torch")
    P = _params(nelx, nely, share)
    out = []
    for variant in (0, 3):
        with Solver(P, precond=EQC_PC_JACOBI, apply_variant=variant) as s:
            out.append(_apply(s, torch, 0))
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("nelx,nely,share", [(1, 1, 1.0), (6, 31, 1.0), (31, 6, 1.0), (32, 7, 0.5), (37, 23, 1.0),
                                             (155, 216, 1.0), (1070, 31, 0.5)])
def test_double_float_apply(eqclib, nelx, nely, share):
    """In double-float arithmetic on small meshes too: the FP64 apply is the slower one there."""
    torch = pytest.importorskip("torch")
    with Solver(_params(nelx, nely, share), precond=EQC_PC_JACOBI) as s:
        y64, ydf = _apply(s, torch, 0), _apply(s, torch, 2)
    assert not np.array_equal(ydf, y64)
    assert np.max(np.abs(ydf - y64)) <= 1e-12 * np.max(np.abs(y64))


@pytest.mark.parametrize("nelx,nely,share", [(13, 15, 1.0), (48, 49, 0.3), (155, 216, 1.0), (156, 217, 0.1)])
def test_residual_of_mixed_solves(eqclib, monkeypatch, nelx, nely, share):
    """As test_residual_of_reliable_updates has it for elements of one rigidity, with its bound of 1e-11."""
    P = _params(nelx, nely, share)
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
