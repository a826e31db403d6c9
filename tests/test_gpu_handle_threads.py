"""One handle per thread: a thread that creates handles does not disturb another one's launches."""
import ctypes as C
import threading

import numpy as np
import pytest

from eqcycle_gb300 import EQC_PC_JACOBI, Solver, preset, set_parameters
from eqcycle_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def test_applies_while_another_thread_creates_handles(eqclib):
    """Launches back to back on a small mesh, where a CTA of the FP64 apply asks for the most shared memory."""
    torch = pytest.importorskip("torch")
    P = set_parameters(preset("homog48").replace(NelX=12, NelY=16, LX=6e3, LY=8e3, creep_depth=6e3))
    stop, errors = threading.Event(), []

    def create():
        try:
            for _ in range(200):
                Solver(P, precond=EQC_PC_JACOBI).close()
        except Exception as e:
            errors.append(e)
        finally:
            stop.set()

    with Solver(P, precond=EQC_PC_JACOBI) as s:
        nx, ny, ld = s.layout()
        x = torch.zeros(ny, ld, dtype=torch.float64)
        x[:, :nx] = torch.as_tensor(np.random.default_rng(3).uniform(-1, 1, (ny, nx)))
        x, y = x.cuda(), torch.zeros(ny, ld, dtype=torch.float64, device="cuda")
        px, py, apply = C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), L.lib().eqc_apply_K_device
        other = threading.Thread(target=create)
        other.start()
        status = set()
        while not stop.is_set():
            for _ in range(500):
                status.add(apply(s.h, px, py, 0))
            status.add(L.lib().eqc_sync(s.h))
        other.join()
        assert status == {0} and not errors
        with Solver(P, precond=EQC_PC_JACOBI, apply_variant=2) as ref:
            z = torch.zeros_like(y)
            L.check(apply(ref.h, px, C.c_void_p(z.data_ptr()), 0), ref.h)
            L.check(L.lib().eqc_sync(ref.h), ref.h)
        assert float((y - z).abs().max()) <= 1e-13 * float(z.abs().max())
