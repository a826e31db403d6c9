"""The FP64 apply is the operator that the caller's derivative matrix H and W define, to rounding.

On a constant field every difference vanishes and K x is what the rounding of H leaves of a derivative of constants,
some 1e-15 of K's entries.  The apply forms it in about 20 roundings per contribution (the row sums of D^T diag(w) D,
the lines' weights, the rigidity, W against mu w_i w_j, the sum at the node), some of them of terms up to ten times
the contribution: 256 eps of the sum of the contributions' sizes is asked.  The same in extended precision, from H
and W as given, is the reference."""
import ctypes as C

import numpy as np
import pytest

from eqcycle_gb300 import EQC_PC_JACOBI, Solver, preset, set_parameters
from eqcycle_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nelx,nely,damage", [(1, 1, 0), (7, 8, 0), (15, 17, 1), (22, 9, 1)])
def test_constant_field(eqclib, nelx, nely, damage):
    torch = pytest.importorskip("torch")
    cfg = preset("dz480").replace(NelX=nelx, NelY=nely, LY=24e3 * nely / nelx, damage=damage, ThickX=12e3, ThickY=9e3)
    P = set_parameters(cfg)
    big = np.longdouble
    H = np.asarray(P.mesh.H).astype(big)
    W = np.asarray(P.mesh.W).transpose(2, 1, 0).reshape(nely, nelx, 5, 5).astype(big)      # [ey, ex, j, i]
    hx, hy = 0.5 * P.mesh.dxe, 0.5 * P.mesh.dye
    one = np.ones((nely, nelx, 5, 5), big)
    row = big(hy / hx) * ((W * (one @ H)) @ H.T)
    col = big(hx / hy) * (H @ (W * (H.T @ one)))
    want, size = (np.zeros((4 * nely + 1, 4 * nelx + 1), big) for _ in range(2))
    for j in range(5):
        for i in range(5):
            at = np.s_[j:j + 4 * nely - 3:4, i:i + 4 * nelx - 3:4]
            want[at] += row[:, :, j, i] + col[:, :, j, i]
            size[at] += abs(row[:, :, j, i]) + abs(col[:, :, j, i])
    with Solver(P, precond=EQC_PC_JACOBI) as s:
        nx, ny, ld = s.layout()
        x = torch.zeros(ny, ld, dtype=torch.float64)
        x[:, :nx] = 1.0
        x, y = x.cuda(), torch.zeros(ny, ld, dtype=torch.float64, device="cuda")
        L.check(L.lib().eqc_apply_K_device(s.h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), 0), s.h)
        L.check(L.lib().eqc_sync(s.h), s.h)
    got = y.cpu().numpy()[:, :nx]
    assert np.all(abs(got - want) <= 256 * np.finfo(np.float64).eps * size.max())
