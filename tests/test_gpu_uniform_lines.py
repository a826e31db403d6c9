"""The FP64 apply's one-contraction lines (k_apply_uni64) against the plain-load kernel, which takes
both contractions of every line: meshes around the edges of its 7 x 8-element tiles, elements of one
rigidity, of several, and both in one tile.

Each result is a sum of at most 4 x 2 lines of some 50 roundings with entries of K's size, so the two
agree to 100 eps of the largest entry of |K| |x|, which max |K x| on random x stands for: 1e-13."""
import ctypes as C

import numpy as np
import pytest

from eqcycle_gb300 import EQC_PC_JACOBI, Solver, preset, set_parameters
from eqcycle_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("material", ["one", "rectangle", "trapezoid", "per-node"])
@pytest.mark.parametrize("nelx,nely", [(1, 1), (1, 9), (6, 7), (7, 8), (8, 9), (13, 15), (14, 16), (15, 17), (63, 65)])
def test_one_contraction_lines_match_two(eqclib, nelx, nely, material):
    torch = pytest.importorskip("torch")
    rule = {"one": 0, "rectangle": 1, "trapezoid": 2, "per-node": 0}[material]
    cfg = preset("dz480").replace(NelX=nelx, NelY=nely, LY=24e3 * nely / nelx, damage=rule, ThickX=12e3, ThickY=9e3)
    P = set_parameters(cfg)
    rng = np.random.default_rng(nelx * 100 + nely)
    if material == "per-node":   # every third element has a rigidity per node
        P.mesh.W[:, :, ::3] *= rng.uniform(0.5, 2.0, P.mesh.W[:, :, ::3].shape)
    out = []
    for variant in (0, 2):
        with Solver(P, precond=EQC_PC_JACOBI, apply_variant=variant) as s:
            nx, ny, ld = s.layout()
            x = torch.zeros(ny, ld, dtype=torch.float64)
            x[:, :nx] = torch.as_tensor(np.random.default_rng(3).uniform(-1, 1, (ny, nx)))
            x, y = x.cuda(), torch.zeros(ny, ld, dtype=torch.float64, device="cuda")
            for _ in range(2):
                L.check(L.lib().eqc_apply_K_device(s.h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), 0), s.h)
            L.check(L.lib().eqc_sync(s.h), s.h)
            out.append(y.cpu().numpy())
    assert not np.any(out[0][:, nx:])            # row padding untouched
    assert np.max(np.abs(out[0] - out[1])) <= 1e-13 * np.max(np.abs(out[1]))
