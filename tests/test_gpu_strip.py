"""The fault strip kernels (k_strip: right-hand side and fault traction of a quasi-static step) at the edges of their
eight element columns: three steps of the plain method, solved to 1e-12, against the oracle's, solved to 1e-13.  Both
are the same arithmetic up to the order of sums and the solvers' stopping, so the states agree to 1e-6, the bound
of the other time-loop comparisons; a wrong column would be off by its own size."""
import numpy as np
import pytest

from eqcycle_gb300 import EQC_FP64, EQC_PC_AMG, Solver, reference_config, set_parameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nelx", [4, 7, 8, 9, 16, 17])
def test_steps_match_oracle(eqclib, oracle_mod, nelx):
    cfg = reference_config(res=1).replace(NelX=nelx, NelY=5)
    P = set_parameters(cfg)
    o = oracle_mod.Oracle(cfg)
    o.run(3, qs_mode=1, qs_tol=1e-13)
    with Solver(P, precision=EQC_FP64, precond=EQC_PC_AMG, cg_tol=1e-12) as s:
        s.init(cfg.V_init)
        st = s.run(3)
        assert st["qs_steps"] == 3
        for k in ("d", "v", "psi", "tau"):
            a, b = s.state(k), o.state(k)
            assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b), k
