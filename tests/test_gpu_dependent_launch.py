"""Steps whose kernels are launched as programmatic dependents.

The step graph overlaps each kernel's first blocks with its predecessor's last
ones; the single-stage calls launch the same kernels one after another. Both
must give the same bits, on either side of the sizes at which the rule
(pdl_pays, csrc/cuda/solver_launch.h) turns the overlap on and off: FP64 2D up
to 53,248 cells (M2AUSM 24,576), 3D up to 8,192, both from 131,072; FP32-bulk at
every size."""
import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu


def _cylinder(nt, nr, ns, solver):
    return cases.cylinder_case(n_theta=nt, n_r=nr, n_span=ns, r1=12, first=0.03, Ls=3, solver=solver, minmod=True,
                               noise=0.02, cfl=0.4)


SHAPES = [(8, 4, 1, 0), (128, 128, 1, 0), (129, 128, 1, 1), (128, 128, 1, 2), (512, 320, 1, 1), (512, 319, 1, 0),
          (32, 16, 16, 1), (33, 16, 16, 1), (32, 16, 16, 2), (64, 32, 24, 0), (64, 33, 24, 1), (64, 48, 38, 1), (64, 64, 32, 1),
          (80, 64, 32, 0), (256, 208, 1, 0), (257, 208, 1, 1), (192, 128, 1, 2), (193, 128, 1, 2), (512, 256, 1, 2),
          (511, 256, 1, 1)]


@pytest.mark.parametrize("precision", [N.LFM_FP64, N.LFM_FP32_BULK])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_step_graph_gives_the_single_stages_bits(shape, precision):
    case = _cylinder(*shape)
    ch = N.CaseHandle.from_case(case)
    a, b = N.Solver(ch, precision=precision), N.Solver(ch, precision=precision)
    steps = 6
    a.step(steps, case.delta_t)
    for _ in range(steps):
        for k in range(5):
            b.stage(k, case.delta_t)
    a.sync()
    b.sync()
    qa, qb = a.get_state(), b.get_state()
    assert np.all(np.isfinite(qa))
    assert np.array_equal(qa, qb)
    # the whole advance as one graph, from page-locked states where torch has them
    q_out = np.empty_like(qa)
    a.advance(ch.q0(), steps, case.delta_t, q_out)
    assert np.array_equal(q_out, qa)
    a.close()
    b.close()
