"""The time step in device memory and the one-launch reductions."""
import numpy as np
import pytest

import oracle.port as P
from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu


def _case(nt, nr, ns=1, solver=1, minmod=True):
    return cases.cylinder_case(n_theta=nt, n_r=nr, n_span=ns, r1=12, first=0.03, Ls=3, solver=solver, minmod=minmod,
                               noise=0.02, cfl=0.4)


@pytest.mark.parametrize("precision", [N.LFM_FP64, N.LFM_FP32_BULK])
@pytest.mark.parametrize("make", [lambda: _case(24, 11), lambda: _case(16, 8, 5), lambda: cases.vortex_case(n=17)],
                         ids=["viscous", "3d", "fused"])
def test_every_step_takes_its_own_dt(make, precision):
    """One graph serves a sequence of time steps, the same as the single
    stages, and the advance graph takes a new dt on the same buffers."""
    case = make()
    ch = N.CaseHandle.from_case(case)
    a, b = N.Solver(ch, precision=precision), N.Solver(ch, precision=precision)
    dts = [case.delta_t * f for f in (1.0, 0.5, 0.5, 0.9, 1.0)]
    for dt in dts:
        a.step(1, dt)
        for k in range(5):
            b.stage(k, dt)
    a.sync()
    b.sync()
    assert np.array_equal(a.get_state(), b.get_state())
    torch = pytest.importorskip("torch")
    q_in, q_out = (torch.empty(ch.q0().shape, dtype=torch.float64, pin_memory=True).numpy() for _ in range(2))
    q_in[...] = ch.q0()
    for dt in (case.delta_t, 0.7 * case.delta_t):
        a.advance(q_in, 3, dt, q_out)
        b.set_state(q_in)
        b.step(3, dt)
        b.sync()
        assert np.array_equal(q_out, b.get_state())
    a.close()
    b.close()


# one block, a block and a cell, many blocks
@pytest.mark.parametrize("shape", [(16, 16, 1), (257, 1, 1), (96, 64, 1), (16, 8, 6)])
def test_reductions_match_the_oracle(shape):
    case = _case(*shape)
    ch = N.CaseHandle.from_case(case)
    s = N.Solver(ch)
    q = ch.q0()
    for _ in range(3):   # the arrival counter resets itself
        assert abs(s.min_dt(0.5) / P.min_dt(ch, q, 0.5) - 1) <= 1e-13
        assert abs(s.cfl(1e-6) / P.cfl(ch, q, 1e-6) - 1) <= 1e-13
    s.close()
