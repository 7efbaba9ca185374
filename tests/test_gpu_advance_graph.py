"""Solver.advance between page-locked states (the whole advance as one graph) gives
the bits of the steps from pageable ones, on either side of the sizes at which
kernels are launched as programmatic dependents (pdl_pays), with a new dt, a new
step count and a new state on the buffers of the first call."""
import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases
from tests.test_gpu_dependent_launch import SHAPES, _cylinder

pytestmark = pytest.mark.gpu


# on either side of the sizes at which FP64 steps change to dependent launches
LINES = [(256, 200, 1, 0), (257, 200, 1, 1), (192, 126, 1, 2), (192, 127, 1, 2), (30, 20, 10, 2), (31, 20, 10, 2),
         (32, 16, 16, 0), (33, 16, 16, 0), (512, 256, 1, 0), (512, 255, 1, 0)]


@pytest.mark.parametrize("precision", [N.LFM_FP64, N.LFM_FP32_BULK])
@pytest.mark.parametrize("shape", [*SHAPES, *LINES, None], ids=lambda s: "x".join(map(str, s)) if s else "vortex")
def test_advance_graph_gives_the_steps_bits(shape, precision):
    torch = pytest.importorskip("torch")
    case = _cylinder(*shape) if shape else cases.vortex_case(n=67, ny=41, solver=0)
    ch = N.CaseHandle.from_case(case)
    a, b = N.Solver(ch, precision=precision), N.Solver(ch, precision=precision)
    q0 = ch.q0()
    q_in, q_out = (torch.empty(q0.shape, dtype=torch.float64, pin_memory=True).numpy() for _ in range(2))
    assert N.load_library().lfm_selftest_kernel_range(q_in.ctypes.data, q_in.nbytes) == 1
    assert N.load_library().lfm_selftest_kernel_range(q_out.ctypes.data, q_out.nbytes) == 1
    for steps, dt, scale in ((3, 1.0, 1.0), (3, 0.5, 1.0), (2, 1.0, 1.001), (3, 1.0, 1.0)):
        q_in[...] = q0 * scale
        q_out[...] = np.nan
        a.advance(q_in, steps, dt * case.delta_t, q_out)
        b.set_state(q0 * scale)      # pageable
        b.step(steps, dt * case.delta_t)
        b.sync()
        assert np.array_equal(q_out, b.get_state())
    a.close()
    b.close()
