"""The FP64 path's own arithmetic against extended precision: reciprocal and
reciprocal root by series, comparisons on the integer pipe, the limiter's and the
pressure polynomials' combined forms. Every bound is counted from the operations
(u = 2^-53, the largest relative error of one)."""
import numpy as np
import pytest

from lfm_public_gb300 import _native as N

pytestmark = pytest.mark.gpu
L = np.longdouble
U = L(2.0) ** -53
TINY, HUGE = np.finfo(np.float64).tiny, np.finfo(np.float64).max


def _values(rng, n, lo, hi):
    """Random mantissas over the exponents lo..hi, the ends of every binade among them."""
    x = rng.uniform(1, 2, n) * 2.0 ** rng.integers(lo, hi + 1, n)
    b = 2.0 ** np.arange(lo, hi + 1, dtype=np.float64)
    return np.concatenate([x, b, np.nextafter(b, 0), np.nextafter(b, np.inf)])


def _ulp(x):
    return np.spacing(np.abs(x)).astype(L)


def test_reciprocal():
    """The series stops at e^3 <= 2^-66: half an ulp and the rounding of a term
    of size 2^-22. Outside binary32's normal range it is the division."""
    x = _values(np.random.default_rng(1), 400000, -124, 122)
    x = np.concatenate([x, -x])
    err = np.abs(N.selftest_fp64("rcp", x).astype(L) * x - 1) * np.abs(1 / x.astype(L))
    assert np.all(err <= L(0.51) * _ulp(1 / x))
    far = _values(np.random.default_rng(2), 20000, -1021, 1022)
    far = far[(far < 2.0 ** -126) | (far > 2.0 ** 126)]
    with np.errstate(divide="ignore", over="ignore"):
        far = np.concatenate([far, -far, [0.0, -0.0, np.inf, -np.inf, TINY, HUGE, TINY / 4, 5e-324]])
        assert np.array_equal(N.selftest_fp64("rcp", far), 1 / far)
    assert np.all(np.isnan(N.selftest_fp64("rcp", np.array([np.nan, -np.nan]))))


def test_reciprocal_root():
    """x y is rounded once before the residual e is formed (u / 2 of the result),
    the series stops at e^3 x 5/16 <= 2^-65, the last operation rounds: at most one
    ulp and a fraction of 2^-12 of it. Outside, CUDA's rsqrt."""
    x = _values(np.random.default_rng(3), 400000, -1021, 1022)
    err = np.abs(N.selftest_fp64("rsqrt", x).astype(L) - 1 / np.sqrt(x.astype(L)))
    inside = (x >= 2.0 ** -125) & (x < 2.0 ** 125)
    ulp = _ulp(1 / np.sqrt(x))
    assert np.all(err[inside] <= L(1.01) * ulp[inside])
    assert np.all(err[~inside] <= 2 * ulp[~inside])
    got = N.selftest_fp64("rsqrt", np.array([0.0, np.inf, -1.0, -1e-300, -np.inf, np.nan]))
    assert got[0] == np.inf and got[1] == 0 and np.all(np.isnan(got[2:]))


def test_comparisons():
    x = _values(np.random.default_rng(4), 20000, -1021, 1023)
    x = np.concatenate([x, -x, [0.0, -0.0, np.inf, -np.inf, 5e-324, -5e-324, HUGE, -HUGE, 1.0, np.nextafter(1, 0)]])
    assert np.array_equal(N.selftest_fp64("pos_part", x), np.where(x < 0, 0.0, x))
    assert np.array_equal(N.selftest_fp64("atleast1", x), (x >= 1).astype(float))
    nan = np.array([np.nan])
    assert np.isnan(N.selftest_fp64("pos_part", nan))[0] and N.selftest_fp64("atleast1", nan)[0] == 0


def _mach_numbers(rng):
    """(M, alpha): all of alpha's range (f_a from 0 to 1), M on both sides of 0, -1
    and 1 down to single ulps."""
    near = np.concatenate([10.0 ** rng.uniform(-16, -1, 4000), [0.0, 2.0 ** -53, 2.0 ** -52]])
    M = np.concatenate([rng.uniform(-1.5, 1.5, 40000), near, -near, 1 - near, 1 + near, -1 + near, -1 - near, [3.0, -3.0, 1e300]])
    fa = rng.uniform(0, 1, M.size)
    fa[::7] = 1.0
    return M, 3 / 16 * (5 * fa * fa - 4)


def test_half_difference_of_the_pressure_polynomials():
    """M (alpha t^2 + 3/4 - M^2 / 4), t = 1 - M^2: t is off by 2 u, its square's term
    by 6 u, the other by 2 u; the sum and the product round once each."""
    M, al = _mach_numbers(np.random.default_rng(5))
    m, a = M.astype(L), al.astype(L)
    inside = np.abs(M) < 1
    with np.errstate(over="ignore"):
        poly = m * (a * (1 - m * m) ** 2 + L(0.75) - m * m / 4)
    ref = np.where(inside, poly, np.sign(m) / 2)
    err = np.abs(N.selftest_fp64("p5half", M, al).astype(L) - ref)
    assert np.all(err <= np.where(inside, 9 * U * np.abs(m) * (L(0.75) + np.abs(a)), 0))
    assert np.all(np.isnan(N.selftest_fp64("p5half", np.array([np.nan]), np.array([0.1]))))


def test_limited_face_values():
    """The reference's limiter (r = 2 gradcf / gradf - 1, held to [0, 1]; beyond a
    quotient of 1000 by sign alone) on the increment it multiplies out to. The two
    products of gradcf round against each other, the face values once."""
    rng = np.random.default_rng(6)
    n = 200000
    P, Q = rng.uniform(-2, 2, (2, n)) * 10.0 ** rng.integers(-6, 6, n)
    Q = np.where(rng.uniform(size=n) < 0.2, P * (1 + 10.0 ** rng.uniform(-16, -8, n)), Q)
    Q[:2000] = P[:2000]
    P[2000:2100], Q[2000:2100] = 1.0e-30, 0.0     # gradf = 0
    d = rng.uniform(-1, 1, (2, n))
    w = rng.uniform(0.2, 0.8, n)
    df = Q - P
    # gradients along d whose quotient lies all over, at 1/2 and 1 to a few ulps, at 1000 and far beyond
    k = rng.uniform(-1.5, 2.5, (2, n)) * np.where(rng.uniform(size=n) < 0.1, 10.0 ** rng.uniform(0, 200, n), 1.0)
    for i, v in enumerate((0.5, 1.0, 1000.0, -1000.0, 0.0)):
        k[:, i::11] = v * (1 + rng.integers(-4, 5, k[:, i::11].shape) * 2.0 ** -52)
    d2 = (d * d).sum(0)
    grads = [k[s] * df * d / d2 for s in (0, 1)]
    grads = [np.where(np.arange(n) % 13 == 0, rng.uniform(-1, 1, (2, n)), g) for g in grads]
    l = lambda x: np.asarray(x).astype(L)  # noqa: E731
    gradf = df + 1.0e-30
    for name, g, side in (("limited_p", grads[0], 1), ("limited_n", grads[1], -1)):
        got = N.selftest_fp64(name, P, Q, grads[0][0], grads[0][1], grads[1][0], grads[1][1], d[0], d[1], w)
        cf = (l(d) * l(g)).sum(0)
        sign = lambda x: np.where(x < 0, L(-1), L(1))  # noqa: E731
        with np.errstate(divide="ignore", invalid="ignore"):
            r = np.where(np.abs(cf) >= 1000 * np.abs(l(gradf)), 2000 * sign(cf) * sign(gradf) - 1, 2 * cf / l(gradf) - 1)
        lim = np.clip(r, 0, 1)
        ref = l(P) + lim * (1 - l(w)) * l(df) if side == 1 else l(Q) - lim * l(w) * l(df)
        # gradcf is off by 2 u of its products' size, which counts where it is not
        # past the quotients that the limiter cuts off; then the limiter by twice
        # that over |gradf| and by 3 roundings of 2 gradcf / gradf (at most 6 u)
        size = np.where(np.abs(cf) <= 2 * np.abs(l(gradf)), np.abs(l(d) * l(g)).sum(0), 0)
        off = np.minimum(4 * U * size + 6 * U * np.abs(l(df)), np.abs(l(df)))
        # its product with the weight (rounded for N's) and the sum
        bound = off + U * (2 * np.abs(l(df)) + np.maximum(np.abs(l(P)), np.abs(l(Q))))
        assert np.all(np.abs(l(got) - ref) <= bound)
