"""Cells with more faces than the fixed-width face tables hold (2D: four).

The FP32-bulk gathers then go through the face lists, in the solver and in the
batch, and a boundary cell's ghosts are found past the tables' width too."""
import numpy as np
import pytest

import oracle.port as P
from lfm_public_gb300 import _native as N, acoustics, cases
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


def merged_case(n, seed, solver, mu):
    """A quad grid with a random half of its cell pairs merged into 2 x 1
    blocks, whose collinear points leave them six faces."""
    rng = np.random.default_rng(seed)
    half, h = 10.0, 20.0 / n
    xs = np.linspace(-half, half, n + 1)
    nodes = np.stack([a.ravel() for a in np.meshgrid(xs, xs, indexing="ij")], axis=1)
    vid = lambda i, j: i * (n + 1) + j  # noqa: E731
    polys = []
    for i in range(0, n, 2):
        for j in range(n):
            a, m, b = vid(i, j), vid(i + 1, j), vid(i + 2, j)
            if rng.uniform() < 0.5:
                polys.append((a, m, b, b + 1, m + 1, a + 1))
            else:
                polys += [(a, m, m + 1, a + 1), (m, b, b + 1, m + 1)]
    case = cases._polygon_mesh(nodes, polys, half, f"merged{n}", solver=solver, n_steps=10, minmod=True)
    case.mu = mu
    case.U_inf = (0.4 * cases.sound_speed(case), 0.0, 0.0)
    case.mach = 0.4
    x, y = case.cell_centres[:, 0], case.cell_centres[:, 1]
    p, T, u, v = cases.isentropic_vortex(case, x, y, 3.0)
    case.fields = {"p": p, "T": T, "U": np.stack([u, v, np.zeros_like(u)], axis=1), "alpha": half - x}
    case.delta_t = cases.acoustic_dt(case, 0.4, np.hypot(u, v), T, np.full(case.n_cells, h))
    return case


@pytest.mark.parametrize("solver,mu", [(0, 0.0), (0, 2.0), (1, 2.0), (2, 0.0), (2, 2.0)])
def test_cells_wider_than_the_tables(solver, mu):
    """FP64 within 1e-12 of the oracle, FP32-bulk p' within 1e-3 of FP64, the
    batch bitwise the single-case solver."""
    case = merged_case(18, 3 + solver, solver, mu)
    ch = N.CaseHandle.from_case(case)
    offs = np.ctypeslib.as_array(ch.desc.cell_face_offsets, shape=(ch.desc.n_cells + 1,))
    assert set(np.diff(offs).tolist()) == {4, 6}
    steps, q = 12, {}
    for prec in (N.LFM_FP64, N.LFM_FP32_BULK):
        s = N.Solver(ch, precision=prec)
        s.step(steps, case.delta_t)
        s.sync()
        q[prec] = s.get_state()
        s.close()
    q_ref, _ = P.run(ch, ch.q0(), steps, case.delta_t)
    assert np.all(rel_l2(q[N.LFM_FP64], q_ref) <= 1e-12), rel_l2(q[N.LFM_FP64], q_ref)
    q32 = q[N.LFM_FP32_BULK]
    assert acoustics.acoustic_rel_l2(q32, q_ref, ch.desc.gamma, case.dim, case.p_inf) <= 1e-3
    b = N.Batch(arena_bytes=N.Batch.case_bytes(ch) + (1 << 20), max_cases=1)
    slot = b.add(ch, case.delta_t)
    b.step(steps)
    b.sync()
    assert np.array_equal(b.get_state(slot), q32)
    b.close()
