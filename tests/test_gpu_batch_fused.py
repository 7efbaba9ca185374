"""Fused batch steps: while every case of a batch is 2D, inviscid and M1 / M2,
a stage is one phase between two primitive buffers; a viscous or 3D case, or
one without current primitives, switches to the separate phases and back. A
case's bits depend on neither."""
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


def _fusable():
    # 32 x 4 = one tile of 128 cells, 129 = a tile and a cell, three triangles' worth of ragged tiles
    cs = [cases.vortex_case(n=32, ny=4, solver=0), cases.vortex_case(n=43, ny=3, solver=1),
          cases.tri_case(n=13, seed=4, solver=1, beta=3.0), cases.vortex_case(n=1, ny=1, solver=0)]
    return cs, [N.CaseHandle.from_case(c) for c in cs]


@pytest.mark.parametrize("shape", [None, (128, 1), (256, 2), (512, 1)])
def test_joining_and_leaving_cases_keep_the_bits(shape):
    """Odd step counts before each change, so that the current primitives sit
    in either buffer when a case joins, leaves or gets a new state."""
    cs, chs = _fusable()
    vis = cases.cylinder_case(n_theta=24, n_r=10, r1=8, first=0.05, Ls=3, solver=2, minmod=True, noise=0.01)
    vh = N.CaseHandle.from_case(vis)
    b = N.Batch(arena_bytes=64 << 20, max_cases=8)
    if shape:
        b.set_tuning(*shape)
    slots = [b.add(h, c.delta_t) for h, c in zip(chs[:3], cs[:3])]
    b.step(3)
    v = b.add(vh, vis.delta_t)          # separate phases from here
    b.step(1)
    last = b.add(chs[3], cs[3].delta_t)
    b.step(3)
    assert np.array_equal(b.get_state(v), _single(vh, 4, vis.delta_t))
    b.remove(v)                          # fused again
    b.step(1)
    b.set_state(slots[1], chs[1].q0())
    b.step(3)
    b.sync()
    steps = [11, 3, 11]
    for s, h, c, n in zip(slots, chs, cs, steps):
        assert np.array_equal(b.get_state(s), _single(h, n, c.delta_t)), c.name
    assert np.array_equal(b.get_state(last), _single(chs[3], 7, cs[3].delta_t))
    b.close()


def test_states_of_many_cases_at_once():
    """More cases than one launch copies (32), with page-locked, pageable and
    absent states side by side: the bits of the separate calls."""
    import torch
    case = cases.vortex_case(n=12, ny=9, solver=0)
    ch = N.CaseHandle.from_case(case)
    n = 37
    a, b = (N.Batch(arena_bytes=n * N.Batch.case_bytes(ch) + (1 << 20), max_cases=n) for _ in range(2))
    sa, sb = [a.add(ch, case.delta_t) for _ in range(n)], [b.add(ch, case.delta_t) for _ in range(n)]
    rng = np.random.default_rng(3)
    q0 = ch.q0()
    states = [q0 * (1 + 1e-3 * rng.uniform(-1, 1, q0.shape)) for _ in range(n)]
    q_in, q_out = [], []
    for k, q in enumerate(states):
        pinned = torch.empty(q.shape, dtype=torch.float64, pin_memory=True).numpy()
        pinned[...] = q
        q_in.append(None if k % 7 == 3 else q if k % 5 == 1 else pinned)
        q_out.append(None if k % 6 == 2 else np.empty_like(q) if k % 4 == 1 else
                     torch.empty(q.shape, dtype=torch.float64, pin_memory=True).numpy())
    for rep in range(2):   # twice: from either primitive buffer
        a.advance(sa, q_in, 3, q_out)
        for k in range(n):
            if q_in[k] is not None:
                b.set_state(sb[k], q_in[k])
        b.step(3)
        b.sync()
        for k in range(n):
            ref = b.get_state(sb[k])
            assert np.array_equal(a.get_state(sa[k]), ref), (rep, k)
            if q_out[k] is not None:
                assert np.array_equal(q_out[k], ref), (rep, k)
    a.close()
    b.close()
