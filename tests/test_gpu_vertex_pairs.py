"""Two smoothing steps of a vertex level in one launch (k_stencil2) against one launch each (EQC_NO_FUSE): the same
bits, on vertex grids around the edges of its 30 x 6-point tiles, for three and four steps (three with the transfer in
one launch, a pair and a single step) in both precisions; the last grid's 40,401 points take the pair in FP64."""
import numpy as np
import pytest

from eqcycle_gb300 import EQC_FP64, EQC_MIXED, EQC_PC_AMG, Solver, preset, set_parameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,variant", [(EQC_FP64, 0), (EQC_MIXED, 8)], ids=["fp64", "mixed"])
@pytest.mark.parametrize("degc", [3, 4])
@pytest.mark.parametrize("nelx,nely", [(29, 23), (30, 24), (31, 29), (59, 36), (200, 200)])
def test_pairs_equal_single_steps(eqclib, monkeypatch, nelx, nely, degc, precision, variant):
    cfg = preset("dz480").replace(NelX=nelx, NelY=nely, LY=24e3 * nely / nelx)
    P = set_parameters(cfg)
    out = []
    for no_fuse in (False, True):
        if no_fuse:
            monkeypatch.setenv("EQC_NO_FUSE", "1")
        with Solver(P, precision=precision, precond=EQC_PC_AMG, apply_variant=variant, mg_degree=3, mg_degree_coarse=degc,
                    mg_coarse_max=64) as s:
            s.init(cfg.V_init)
            st = s.run(4)
            out.append((st["cg_iters"], {k: s.state(k) for k in ("d", "v", "psi", "tau")}))
    assert out[0][0] == out[1][0] > 0
    for k in out[0][1]:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
