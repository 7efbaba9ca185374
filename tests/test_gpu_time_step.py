"""The time step in device memory, the one-launch reductions, and the residual's
one-launch preparation."""
import ctypes as C

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


@pytest.mark.parametrize("precision", [N.LFM_FP64, N.LFM_FP32_BULK])
@pytest.mark.parametrize("shape", [(24, 11, 1), (16, 8, 5)])
def test_residual_after_other_contents_of_the_scratch(shape, precision):
    """M2AUSM without minmod reads zero gradients in every cell and ghost: the
    scratch array still holds the previous call's. Also replayed from a graph."""
    torch = pytest.importorskip("torch")
    lib = N.load_library()
    got = {}
    stream = torch.cuda.Stream()
    for minmod in (True, False, True, False):
        case = _case(*shape, solver=2, minmod=minmod)
        case.residuals = True   # the oracle records them then
        ch = N.CaseHandle.from_case(case)
        s = N.Solver(ch, precision=precision)
        q = torch.from_numpy(ch.q0()).to("cuda")
        res = torch.full_like(q, float("nan"))
        torch.cuda.synchronize()
        call = lambda: N.check(lib.lfm_solver_residual_noalloc(  # noqa: E731
            s._h, C.c_void_p(q.data_ptr()), q.shape[1], C.c_void_p(res.data_ptr()), C.c_void_p(stream.cuda_stream)))
        call()
        stream.synchronize()
        first = res.cpu().numpy()
        _, expected = P.cell_residual(ch, ch.q0(), 1, case.delta_t)
        scale = np.abs(expected).max(axis=1, keepdims=True)
        assert np.max(np.abs(first - expected) / scale) <= (1e-11 if precision == N.LFM_FP64 else 1e-4)
        assert np.array_equal(got.setdefault(minmod, first), first)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            call()
        res.fill_(float("nan"))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(res.cpu().numpy(), first)
        s.close()
