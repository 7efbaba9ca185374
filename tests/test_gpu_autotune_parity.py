"""Autotuning between steps keeps the bits of the steps after it, also where the
stages alternate two primitive buffers and the current one is the second."""
import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", [1, 2, 3])
@pytest.mark.parametrize("form", ["fused", "viscous", "tiles"])
def test_steps_around_an_autotune(monkeypatch, form, before):
    if form == "tiles":
        monkeypatch.setenv("LFM_TILE_CELLS", "128")
    if form == "fused":
        case = cases.vortex_case(n=37, ny=29, solver=1)
    else:
        case = cases.cylinder_case(n_theta=40, n_r=17, r1=8, first=0.05, solver=0, noise=0.01)
    ch = N.CaseHandle.from_case(case)
    a, b = (N.Solver(ch, precision=N.LFM_FP32_BULK) for _ in range(2))
    a.step(before, case.delta_t)
    a.autotune(case.delta_t, trial_steps=2, flush_bytes=1 << 20)
    a.step(3, case.delta_t)
    b.step(before + 3, case.delta_t)
    a.sync()
    b.sync()
    assert np.array_equal(a.get_state(), b.get_state())
    a.close()
    b.close()
