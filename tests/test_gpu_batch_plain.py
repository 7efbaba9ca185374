"""Phases of batches without M2AUSM and without cells wider than the fixed-width
tables run kernels of their own; a case that has either switches the batch to
the general ones and back. A case's bits depend on neither."""
import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu


def _single(ch, n, dt):
    s = N.Solver(ch, precision=N.LFM_FP32_BULK)
    s.step(n, dt)
    s.sync()
    q = s.get_state()
    s.close()
    return q


def _cyl(nt, nr, ns, solver):
    return cases.cylinder_case(n_theta=nt, n_r=nr, n_span=ns, r1=8, first=0.05, Ls=3, solver=solver, minmod=True,
                               noise=0.01)


@pytest.mark.parametrize("shape", [None, (128, 1, 0, 1, 1), (256, 2, 1, 1, 1), (512, 1, 0, 1, 1), (128, 1, 0, 1, 0)])
@pytest.mark.parametrize("dims", [2, 3])
def test_plain_and_general_phases_give_the_same_bits(dims, shape):
    cs = [_cyl(24, 10, 1, 0), _cyl(33, 17, 1, 1), cases.vortex_case(n=19, solver=1)]
    if dims == 3:
        cs += [_cyl(16, 9, 5, 1), _cyl(13, 8, 4, 0)]
    chs = [N.CaseHandle.from_case(c) for c in cs]
    ausm = _cyl(21, 9, 3 if dims == 3 else 1, 2)
    ah = N.CaseHandle.from_case(ausm)
    b = N.Batch(arena_bytes=64 << 20, max_cases=8)
    if shape:
        b.set_tuning(*shape)
    slots = [b.add(h, c.delta_t) for h, c in zip(chs, cs)]
    b.step(3)
    a = b.add(ah, ausm.delta_t)          # general from here
    b.step(2)
    assert np.array_equal(b.get_state(a), _single(ah, 2, ausm.delta_t))
    b.remove(a)                          # plain again
    b.step(2)
    b.sync()
    for s, h, c in zip(slots, chs, cs):
        assert np.array_equal(b.get_state(s), _single(h, 7, c.delta_t)), c.name
    b.close()


def test_launches_per_step():
    """Fused stages are one kernel, phased ones one per phase, persistent ones one."""
    vortex, viscous = cases.vortex_case(n=9, solver=0), _cyl(12, 8, 1, 0)
    vh, ch = N.CaseHandle.from_case(vortex), N.CaseHandle.from_case(viscous)
    b = N.Batch(arena_bytes=16 << 20, max_cases=4)
    b.add(vh, vortex.delta_t)
    assert b.launches_per_step() == 5
    s = b.add(ch, viscous.delta_t)
    assert b.launches_per_step() == 15
    b.remove(s)
    b.set_tuning(128, 1, 0, 1, 1)
    assert b.launches_per_step() == 10
    b.set_tuning(128, 1, 0, 1, 0)
    assert b.launches_per_step() == 5
    b.close()
