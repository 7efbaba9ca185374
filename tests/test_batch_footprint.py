"""Footprint of a case in a batch (lfm_batch_case_bytes): callers size arenas by it,
so no case outgrows the block it took with its values in rows of single values
and one primitive buffer -- strips with more ghosts than cells included."""
import pytest

from lfm_public_gb300 import _native as N, cases


def _cyl(nt, nr, ns, solver):
    return cases.cylinder_case(n_theta=nt, n_r=nr, n_span=ns, r1=8, first=0.05, Ls=3, solver=solver, minmod=True)


LIMITS = [(cases.vortex_case, dict(n=1, ny=1, solver=0), 6400), (cases.vortex_case, dict(n=1, ny=8, solver=0), 7936),
          (cases.vortex_case, dict(n=200, ny=1, solver=0), 102912), (cases.vortex_case, dict(n=400, ny=2, solver=0), 314880),
          (cases.vortex_case, dict(n=3000, ny=1, solver=0), 1490944), (cases.vortex_case, dict(n=64, ny=64, solver=0), 1186816),
          (cases.tri_case, dict(n=1, seed=1, solver=1), 6400), (cases.tri_case, dict(n=40, seed=1, solver=1), 789248),
          (_cyl, dict(nt=24, nr=10, ns=1, solver=2), 92672), (_cyl, dict(nt=300, nr=1, ns=1, solver=1), 181760),
          (_cyl, dict(nt=16, nr=9, ns=5, solver=1), 404480), (_cyl, dict(nt=40, nr=1, ns=40, solver=2), 1730048),
          (_cyl, dict(nt=300, nr=1, ns=2, solver=1), 544000)]


@pytest.mark.parametrize("make,kw,limit", LIMITS)
def test_no_case_outgrows_its_block(make, kw, limit):
    assert N.Batch.case_bytes(N.CaseHandle.from_case(make(**kw))) <= limit
