"""The bounded grid-barrier wait (failure detection on the host, no GPU fault) in a
batch whose launch shape nobody chose: the persistent kernel runs while a barrier
is made to wait, and the default launches again afterwards."""
import time

import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("viscous", [False, True])
def test_default_batch_reports_a_barrier_that_gave_up(viscous):
    case = (cases.cylinder_case(n_theta=24, n_r=10, r1=8, first=0.05, solver=0, noise=0.01) if viscous
            else cases.vortex_case(n=32, solver=1))
    ch = N.CaseHandle.from_case(case)

    def batch():
        b = N.Batch(arena_bytes=N.Batch.case_bytes(ch) + (1 << 20), max_cases=1)
        return b, b.add(ch, case.delta_t)

    b, _ = batch()
    b.debug_barrier(1)
    assert b.launches_per_step() == 5
    t0 = time.perf_counter()
    b.step(1)
    with pytest.raises(N.LfmError) as e:
        b.sync()
    b.close()
    assert e.value.code == N.LFM_ERR_CUDA and "barrier" in str(e.value)
    assert time.perf_counter() - t0 < 20.0
    # given and taken back before a step: the default launches, the same bits
    (b, slot), (c, ref) = batch(), batch()
    b.debug_barrier(1)
    b.debug_barrier(0)
    assert b.launches_per_step() == c.launches_per_step()
    b.step(3)
    c.step(3)
    b.sync()
    c.sync()
    assert np.array_equal(b.get_state(slot), c.get_state(ref))
    b.close()
    c.close()
    # phased launches that were asked for have no barrier
    b, slot = batch()
    b.set_tuning(128, 1, 0, 1, 1)
    b.debug_barrier(1)
    b.step(3)
    b.sync()
    b.close()
