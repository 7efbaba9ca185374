"""Batch.advance with a slot or an output buffer listed more than once: the last
entry wins, as in the separate calls, whatever memory the states are in."""
import itertools

import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu


def _array(shape, pinned):
    torch = pytest.importorskip("torch")
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy() if pinned else np.empty(shape)


def _states(ch, n):
    rng = np.random.default_rng(5)
    return [ch.q0() * (1 + 1e-3 * rng.uniform(-1, 1, ch.q0().shape)) for _ in range(n)]


def _batch(ch, dt, n):
    b = N.Batch(arena_bytes=n * N.Batch.case_bytes(ch) + (1 << 20), max_cases=n)
    return b, [b.add(ch, dt) for _ in range(n)]


@pytest.mark.parametrize("pinned", list(itertools.product([True, False], repeat=3)))
@pytest.mark.parametrize("steps", [0, 3])
def test_slot_given_several_states(pinned, steps):
    case = cases.vortex_case(n=251, ny=173, solver=0)   # many blocks a state
    ch = N.CaseHandle.from_case(case)
    (a, sa), (b, sb) = _batch(ch, case.delta_t, 2), _batch(ch, case.delta_t, 2)
    states = _states(ch, 4)
    order = [0, 0, 1, 0]   # slot 0 three times, slot 1 between
    for rep in range(3):
        q_in = [_array(q.shape, p) for q, p in zip(states, (*pinned[:2], True, pinned[2]))]
        for dst, q in zip(q_in, states):
            dst[...] = q
        out = [np.empty_like(states[0]) for _ in sa]
        a.advance([sa[k] for k in order] + sa, q_in + [None, None], steps, [None] * 4 + out)
        for k, q in zip(order, states):
            b.set_state(sb[k], q)
        b.step(steps)
        b.sync()
        for o, s in zip(out, sb):
            assert np.array_equal(o, b.get_state(s)), rep
    a.close()
    b.close()


@pytest.mark.parametrize("pinned", [True, False])
def test_output_buffer_of_several_slots(pinned):
    case = cases.vortex_case(n=251, ny=173, solver=0)
    ch = N.CaseHandle.from_case(case)
    b, slots = _batch(ch, case.delta_t, 3)
    states = _states(ch, 3)
    for s, q in zip(slots, states):
        b.set_state(s, q)
    refs = [b.get_state(s) for s in slots]
    out, other = _array(refs[0].shape, pinned), _array(refs[0].shape, pinned)
    for order in itertools.permutations(range(3)):
        b.advance([slots[k] for k in order], None, 0, [out, other, out])
        assert np.array_equal(out, refs[order[2]])
        assert np.array_equal(other, refs[order[1]])
    # two states that overlap by all but one row: the later entry's rows stand
    nq, nc = refs[0].shape
    flat = _array(((nq + 1) * nc,), pinned)
    first, second = flat[:nq * nc].reshape(nq, nc), flat[nc:].reshape(nq, nc)
    b.advance(slots[:2], None, 0, [first, second])
    assert np.array_equal(first[0], refs[0][0]) and np.array_equal(second, refs[1])
    b.advance(slots[:2], None, 0, [second, first])
    assert np.array_equal(first, refs[1]) and np.array_equal(second[-1], refs[0][-1])
    b.close()
