"""The learned guess's loss is a sum in FP64: squares below and above FP32's range count in full.

A network of zeros gives zero outputs, so the loss is the targets' mean square: each square exact but for one
rounding, the sums of 7,381 entries and of the batch within sqrt(1e6) eps = 2e-13 of it; 1e-12 is asked."""
import numpy as np
import pytest

from eqcycle_gb300 import EQC_PC_JACOBI, Solver, preset, set_parameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-25, 1.0, 1e19])
@pytest.mark.parametrize("batch", [1, 5, 65])
def test_loss_over_the_range_of_targets(eqclib, batch, scale):
    P = set_parameters(preset("homog48").replace(NelX=13, NelY=4, LX=6.5e3, LY=2e3, creep_depth=6.5e3))
    rng = np.random.default_rng(batch)
    with Solver(P, precond=EQC_PC_JACOBI) as s:
        nin, nout, npar = s.guess_shape()
        s.set_guess_params(np.zeros(npar, np.float32))
        x0 = rng.uniform(-1, 1, (batch, nin)).astype(np.float32)
        tgt = (scale * rng.uniform(-1, 1, (batch, nout))).astype(np.float32)
        loss = s.guess_grad(x0, tgt)[1]
        mse = s.guess_eval(x0, tgt)
    want = float(np.mean(tgt.astype(np.longdouble) ** 2))
    assert abs(loss - want) <= 1e-12 * want and abs(mse - want) <= 1e-12 * want


def test_gradient_allocates_nothing_of_its_own(eqclib):
    """After an evaluation of as many pairs the buffers of a batch are there: a handle's first gradient takes no more
    device memory (its kernels loaded by another handle's)."""
    torch = pytest.importorskip("torch")
    P = set_parameters(preset("homog48").replace(NelX=13, NelY=4, LX=6.5e3, LY=2e3, creep_depth=6.5e3))
    rng = np.random.default_rng(1)
    with Solver(P, precond=EQC_PC_JACOBI) as other, Solver(P, precond=EQC_PC_JACOBI) as s:
        nin, nout, _ = s.guess_shape()
        x0 = rng.uniform(-1, 1, (65, nin)).astype(np.float32)
        tgt = rng.uniform(-1, 1, (65, nout)).astype(np.float32)
        other.guess_grad(x0, tgt)
        s.guess_eval(x0, tgt)
        free = torch.cuda.mem_get_info()[0]
        s.guess_grad(x0, tgt)
        assert torch.cuda.mem_get_info()[0] == free
