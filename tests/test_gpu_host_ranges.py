"""States in page-locked memory are read and written by kernels where they lie
only if they are aligned for doubles and page-locked to their end; any other
state goes through the copy calls, with the same bits."""
import ctypes as C

import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu


def test_range_decision():
    """Queries only: nothing at these addresses is accessed."""
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    direct = N.load_library().lfm_selftest_kernel_range
    a = np.zeros(4 << 20, dtype=np.uint8)
    page, mb = 1 << 16, 1 << 20
    base = (a.ctypes.data + page - 1) // page * page
    assert direct(C.c_void_p(base), 64) == 0                      # pageable
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(base, mb, 0)) == 0
    assert int(rt.cudaHostRegister(base + 2 * mb, mb, 0)) == 0    # 1 MB between the two is pageable
    try:
        assert direct(C.c_void_p(base), mb) == 1
        assert direct(C.c_void_p(base + mb - 8), 8) == 1
        assert direct(C.c_void_p(base), mb + 8) == 0              # past the registration's end
        assert direct(C.c_void_p(base + mb - 8), 16) == 0
        assert direct(C.c_void_p(base), 3 * mb) == 0              # first and last byte page-locked, not all between
        assert direct(C.c_void_p(base + mb), 8) == 0
        for off in range(1, 8):
            assert direct(C.c_void_p(base + off), 64) == 0        # not aligned for doubles
    finally:
        assert int(rt.cudaHostUnregister(base)) == 0
        assert int(rt.cudaHostUnregister(base + 2 * mb)) == 0
    assert direct(C.c_void_p(base), 64) == 0


def _pinned(shape, offset=0):
    """Page-locked float64 array whose address is `offset` bytes past an aligned one."""
    torch = pytest.importorskip("torch")
    n = 8 * int(np.prod(shape))
    return torch.empty(n + 16, dtype=torch.uint8, pin_memory=True).numpy()[offset:offset + n].view(np.float64).reshape(shape)


@pytest.mark.parametrize("offset", [4, 1])
@pytest.mark.parametrize("precision", [N.LFM_FP64, N.LFM_FP32_BULK])
def test_misaligned_states_of_a_solver(precision, offset):
    case = cases.vortex_case(n=19, ny=13, solver=1)
    ch = N.CaseHandle.from_case(case)
    s = N.Solver(ch, precision=precision)
    q0 = ch.q0()
    ref = np.empty_like(q0)
    s.advance(q0, 3, case.delta_t, ref)
    for oin, oout in ((offset, offset), (0, offset), (offset, 0), (0, 0)):
        q_in, q_out = _pinned(q0.shape, oin), _pinned(q0.shape, oout)
        q_in[...] = q0
        s.advance(q_in, 3, case.delta_t, q_out)
        assert np.array_equal(q_out, ref)
        s.set_state(q_in)
        s.step(3, case.delta_t)
        s.sync()
        q_out[...] = 0
        s.get_state(q_out)
        assert np.array_equal(q_out, ref)
    s.close()


def test_misaligned_states_of_a_batch():
    case = cases.vortex_case(n=19, ny=13, solver=1)
    ch = N.CaseHandle.from_case(case)
    q0 = ch.q0()
    b = N.Batch(arena_bytes=4 * N.Batch.case_bytes(ch) + (1 << 20), max_cases=4)
    slots = [b.add(ch, case.delta_t) for _ in range(4)]
    b.step(3)
    ref = b.get_state(slots[0])
    q_in, q_out = [_pinned(q0.shape, o) for o in (4, 0, 1, 4)], [_pinned(q0.shape, o) for o in (0, 4, 1, 4)]
    for q in q_in:
        q[...] = q0
    b.advance(slots, q_in, 3, q_out)
    for q in q_out:
        assert np.array_equal(q, ref)
    b.set_state(slots[1], q_in[0])
    b.step(3)
    b.sync()
    out = _pinned(q0.shape, 4)
    b.get_state(slots[1], out)
    assert np.array_equal(out, ref)
    b.close()
