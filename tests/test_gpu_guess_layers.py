"""The learned guess's layers as tiled FP32 products (gemm32.cuh) at the edges of their 64 x 64 x 16 tiles, of the
batch below which small kernels run (4), and of the splits of long sums over a cluster: network outputs, loss and
every parameter block's gradient against the CPU restatement in 64 bits.

Up to twelve products in a chain of at most 7,381 terms each: relative rounding errors of sqrt(7381) 2^-24 = 5e-6 a
product, 2e-5 for the chain; a gradient block's norm may be a few times smaller than its terms', so 1e-4 as for the
small batch of test_learned_guess.py."""
import numpy as np
import pytest

from eqcycle_gb300 import EQC_PC_JACOBI, Solver, preset, set_parameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nelx,batch", [(1, 1), (1, 5), (4, 64), (12, 4), (13, 65), (16, 17), (31, 129), (33, 6), (64, 260)])
def test_layers_match_restatement(eqclib, nelx, batch):
    from oracle import guessnet as gn
    P = set_parameters(preset("homog48").replace(NelX=nelx, NelY=4, LX=500.0 * nelx, LY=2e3, creep_depth=500.0 * nelx))
    rng = np.random.default_rng(nelx * 1000 + batch)
    with Solver(P, precond=EQC_PC_JACOBI) as s:
        nin, nout, npar = s.guess_shape()
        p = (rng.uniform(-1, 1, npar) * 0.1).astype(np.float32)
        s.set_guess_params(p)
        x0 = rng.uniform(-1, 1, (batch, nin)).astype(np.float32)
        tgt = rng.uniform(-1, 1, (batch, nout)).astype(np.float32)
        g, loss = s.guess_grad(x0, tgt)
        g2, loss2 = s.guess_grad(x0, tgt)
        mse, out = s.guess_eval(x0, tgt, outputs=True)
    assert np.array_equal(g, g2) and loss == loss2   # fixed orders of summation
    ref_loss, g_ref, out_ref = gn.loss_and_grad(p.astype(np.float64), x0, tgt)

    def rel(a, b):
        return float(np.linalg.norm(a - b) / np.linalg.norm(b))

    assert rel(out, out_ref) <= 2e-5
    assert abs(loss - ref_loss) <= 2e-5 * ref_loss and abs(mse - ref_loss) <= 2e-5 * ref_loss
    for name, (o, shp) in gn.shapes(P.int_.FltNglob)[2].items():
        k = int(np.prod(shp))
        assert rel(g[o:o + k], g_ref[o:o + k]) <= 1e-4, name
