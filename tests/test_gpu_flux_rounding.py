"""Rounding of a face's FP64 flux.

Momentum: the viscous sum rounds at its own size and joins the pressure term p S
in one operation. The state makes everything else exact: density 1, gamma 1.5, R 1, weights 1/2,
pressures and velocities of few bits, so that the primitives and the face values
carry no rounding, and viscous and convective terms below 1 % of p S, so that
theirs does not count. With p S in one binade, [1/2, 1), a momentum residual on
the quads then has the rounding of its two faces' p S -- one operation each, at
most three where the product, the convective and the viscous term were rounded one
after another -- and at most two of the sum over the faces: not above 8 roundings
of a uniform error of variance ulp^2 / 12. One operation a viscous term would make
it 14.

Energy, M1: the mass flux times gamma / (gamma - 1) R psi holds the reciprocal of
the density once, in R psi. The state gives every cell one density whose
reciprocal rounds by almost half an ulp, delta <= u = 2^-53, and makes the rest of
the primitives exact but for one product. What rounds then, at the size of the
flux: that product (two cells' mean, half the variance), the interpolated R psi,
the mass flux, and at most three operations to the energy flux, each of variance at
most u^2 / 3; the sum over the faces three more. So the residual is off by at most
sqrt(1 + 8.5 / 3) u, 1.96 u, of its size, and delta twice, with an operation more,
would be sqrt(4 + 9.5 / 3 x 1/2) u, 2.36 u, even at half of each variance."""
import ctypes as C

import numpy as np
import pytest

from lfm_public_gb300 import _native as N, cases

pytestmark = pytest.mark.gpu
MU, GAMMA = 2.0 ** -8, 1.5


def _view(p, n):
    return np.ctypeslib.as_array(p, shape=(n,))


def _case(solver, n, mu=MU, rho=1.0):
    case = cases.vortex_case(n=n, solver=solver, mu=mu)
    ch = N.CaseHandle.from_case(case)
    d = ch.desc
    d.gamma, d.Rgas = GAMMA, 1.0
    _view(d.w, d.n_faces)[:] = 0.5
    rng = np.random.default_rng(11)
    nc = d.n_cells
    face = np.abs(_view(d.S, 2 * d.n_faces)).max()   # every face has this area
    p = np.round(rng.uniform(0.52, 0.98, nc) / face * 2.0 ** 20) * 2.0 ** -20
    u = rng.integers(-200, 201, (2, nc)) * 2.0 ** -12
    q = np.stack([np.full(nc, rho), *(rho * u), p / (GAMMA - 1) + 0.5 * rho * (u * u).sum(0)])
    assert np.array_equal((GAMMA - 1) * (q[3] - 0.5 * (q[1] * u[0] + q[2] * u[1])), p)
    return ch, q, u, p


def _momentum_residual(d, q, u, p, solver):
    """In extended precision; also which cells have no ghost among their
    neighbours' neighbours."""
    L = np.longdouble
    nc, nf = d.n_cells, d.n_faces
    P, Q = _view(d.face_p, nf), _view(d.face_n, nf)
    S, K = (_view(a, 2 * nf).reshape(2, nf).astype(L) for a in (d.S, d.K))
    lap = _view(d.delta_mag, nf).astype(L) * _view(d.dmag_inv, nf).astype(L)
    vi = _view(d.vol_inv, nc).astype(L)
    inner = Q < nc

    def scatter(x):
        out = np.zeros(nc, L)
        np.add.at(out, P, x)
        np.add.at(out, Q[inner], -x[inner])
        return out

    u, p = (np.concatenate([a.astype(L), np.zeros((*a.shape[:-1], d.n_ghosts), L)], -1) for a in (u, p))
    half = L(0.5)
    mid = lambda x: half * (x[..., P] + x[..., Q])  # noqa: E731
    grad = np.zeros((2, 2, nc + d.n_ghosts), L)
    for a in range(2):
        for b in range(2):
            grad[a, b, :nc] = scatter(mid(u[a]) * S[b]) * vi
    g, uf = mid(grad), mid(u)
    phi = (uf * S).sum(0)
    mu, tr = L(MU), g[0, 0] + g[1, 1]
    res = []
    for x in range(2):
        vis = mu * ((g[:, x] * S).sum(0) - L(2) / 3 * tr * S[x] + lap * (u[x][Q] - u[x][P]) + (K * g[x]).sum(0))
        res.append(scatter(vis - uf[x] * phi - mid(p) * S[x]))
    near = np.zeros(nc, bool)
    near[P[~inner]] = True
    for _ in range(2):
        grown = near.copy()
        grown[P[inner & near[np.minimum(Q, nc - 1)]]] = True
        grown[Q[inner & near[P]]] = True
        near = grown
    return np.stack(res), ~near


def _residual(ch, q):
    torch = pytest.importorskip("torch")
    s = N.Solver(ch, precision=N.LFM_FP64)
    qd = torch.from_numpy(q).cuda()
    res = torch.empty_like(qd)
    N.check(N.load_library().lfm_solver_residual_noalloc(s._h, C.c_void_p(qd.data_ptr()), q.shape[1],
                                                         C.c_void_p(res.data_ptr()), None))
    torch.cuda.synchronize()
    s.close()
    return res.cpu().numpy()


@pytest.mark.parametrize("solver", [0, 1])
@pytest.mark.parametrize("n", [50, 93])
def test_viscous_terms_round_at_their_own_size(solver, n):
    ch, q, u, p = _case(solver, n)
    ref, deep = _momentum_residual(ch.desc, q, u, p, solver)
    assert deep.sum() > 1000
    err = (_residual(ch, q)[1:3] - ref)[:, deep].astype(np.float64)
    ulp = 2.0 ** -53   # of [1/2, 1)
    rms = np.sqrt((err * err).mean(axis=1)) / ulp
    assert np.all(rms <= np.sqrt(8 / 12)), rms


@pytest.mark.parametrize("n", [50, 93])
def test_energy_flux_of_m1_holds_the_density_once(n):
    L = np.longdouble
    # few bits, below 1: the reciprocal's error is largest just above 1
    rhos = 1 - np.arange(1, 256) * 2.0 ** -12
    delta = np.abs((L(1) / rhos - (1 / rhos)) * rhos)
    rho = float(rhos[np.argmax(delta)])
    assert delta.max() > 0.95 * 2.0 ** -53
    ch, q, u, p = _case(0, n, 0.0, rho)
    d = ch.desc
    P, Q = _view(d.face_p, d.n_faces), _view(d.face_n, d.n_faces)
    S = _view(d.S, 2 * d.n_faces).reshape(2, -1).astype(L)
    inner = Q < d.n_cells
    P, Q, S, bound = P[inner], Q[inner], S[:, inner], P[~inner]
    m, R = q[1:3].astype(L), p.astype(L) / rho
    mf, Rf = (m[:, P] + m[:, Q]) / 2, (R[P] + R[Q]) / 2
    flux = (mf * S).sum(0) * (L(GAMMA) / (L(GAMMA) - 1) * Rf + (mf * mf).sum(0) / (2 * L(rho) ** 2))
    ref = np.zeros(d.n_cells, L)
    np.add.at(ref, P, -flux)
    np.add.at(ref, Q, flux)
    deep = np.ones(d.n_cells, bool)
    deep[bound] = False
    err = (_residual(ch, q)[3] - ref)[deep].astype(np.float64)
    off = np.sqrt((err * err).mean() / (ref[deep].astype(np.float64) ** 2).mean()) * 2.0 ** 53
    assert off <= np.sqrt(1 + 8.5 / 3), off
