"""A batch without cases steps, advances and is timed without effect, in every
launch shape, before its first case joins and after its last one has left."""
import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu


def _cylinder(solver):
    return cases.cylinder_case(n_theta=24, n_r=10, r1=8, first=0.05, solver=solver, minmod=True, noise=0.01)


def _single(ch, n, dt):
    s = N.Solver(ch, precision=N.LFM_FP32_BULK)
    s.step(n, dt)
    s.sync()
    q = s.get_state()
    s.close()
    return q


@pytest.mark.parametrize("make", [lambda: cases.vortex_case(n=21, solver=0), lambda: _cylinder(0), lambda: _cylinder(2)],
                         ids=["fused", "phased", "ausm"])
@pytest.mark.parametrize("shape", [None, (128, 1, 0, 1, 0), (256, 2, 1, 0, 0), (512, 1, 0, 1, 1)])
def test_empty_batch_steps(make, shape):
    case = make()
    ch = N.CaseHandle.from_case(case)
    b = N.Batch(arena_bytes=2 * N.Batch.case_bytes(ch) + (1 << 20), max_cases=2)
    if shape:
        b.set_tuning(*shape)

    def empty():
        for n in (0, 1, 3):
            b.step(n)
        b.sync()
        b.advance([], [], 2, [])
        assert len(b.bench(2)) == 2

    empty()
    for rep in range(2):
        slot = b.add(ch, case.delta_t)
        b.step(3)
        assert np.array_equal(b.get_state(slot), _single(ch, 3, case.delta_t)), rep
        b.remove(slot)
        empty()
    b.close()


def test_empty_batch_autotunes():
    case = cases.vortex_case(n=21, solver=1)
    ch = N.CaseHandle.from_case(case)
    b = N.Batch(arena_bytes=N.Batch.case_bytes(ch) + (1 << 20), max_cases=1)
    b.autotune(1)
    slot = b.add(ch, case.delta_t)
    b.step(2)
    assert np.array_equal(b.get_state(slot), _single(ch, 2, case.delta_t))
    b.close()
