"""Descriptions in which several faces of one cell share a boundary ghost: a cell's
ghosts are found whatever their numbers, and the bits are those of a ghost a
face (the ghosts are walls, whose state is the cell's own, mirrored)."""
import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases
from tests.test_gpu_wide_cells import merged_case

pytestmark = pytest.mark.gpu

# per position among a cell's boundary faces, the position whose ghost it takes
PATTERNS = {"first_third": (0, 1, 0, 3, 4), "first_second": (0, 0, 2, 3, 4), "second_third": (0, 1, 1, 3, 4),
            "all": (0, 0, 0, 0, 0), "two_pairs": (0, 1, 0, 1, 0), "own": (0, 1, 2, 3, 4)}


def _description(make, pattern):
    case = make()
    ch = N.CaseHandle.from_case(case)
    d = ch.desc
    kind = np.ctypeslib.as_array(d.ghost_kind, shape=(d.n_ghosts,))
    face_p = np.ctypeslib.as_array(d.face_p, shape=(d.n_faces,))
    face_n = np.ctypeslib.as_array(d.face_n, shape=(d.n_faces,))
    kind[:] = 1
    widest = 0
    for c in np.unique(face_p[face_n >= d.n_cells]):
        faces = np.flatnonzero((face_p == c) & (face_n >= d.n_cells))
        ghosts = face_n[faces].copy()
        widest = max(widest, len(faces))
        for k, f in enumerate(faces):
            face_n[f] = ghosts[min(PATTERNS[pattern][k], len(ghosts) - 1)]
    return case, ch, widest


MESHES = {"one_cell": lambda: cases.vortex_case(n=1, ny=1, solver=0), "strip": lambda: cases.vortex_case(n=1, ny=5, solver=1),
          "viscous_strip": lambda: cases.vortex_case(n=1, ny=5, solver=1, mu=1.0),
          "wide": lambda: merged_case(4, 3, 0, 0.0), "wide_viscous": lambda: merged_case(2, 2, 1, 2.0)}


def _states(case, ch):
    out = []
    for prec in (N.LFM_FP64, N.LFM_FP32_BULK):
        s = N.Solver(ch, precision=prec)
        s.step(3, case.delta_t)
        s.sync()
        out.append(s.get_state())
        s.close()
    b = N.Batch(arena_bytes=N.Batch.case_bytes(ch) + (1 << 20), max_cases=1)
    slot = b.add(ch, case.delta_t)
    b.step(3)
    b.sync()
    out.append(b.get_state(slot))
    b.close()
    return out


@pytest.mark.parametrize("mesh", list(MESHES))
def test_faces_that_share_a_ghost(mesh):
    case, ch, widest = _description(MESHES[mesh], "own")
    assert widest >= 3
    refs = _states(case, ch)
    assert all(np.all(np.isfinite(q)) for q in refs)
    for pattern in PATTERNS:
        case, ch, _ = _description(MESHES[mesh], pattern)
        for q, ref in zip(_states(case, ch), refs):
            assert np.array_equal(q, ref), pattern
