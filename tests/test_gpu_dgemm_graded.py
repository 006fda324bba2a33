"""mq_dgemm where the elements of a row or column differ by many orders of magnitude
and the large ones meet zeros, so that a bound by the rows' norms says nothing.

Bound per element, with t = sum |a||b| of its own products: K roundings of an FP64 sum
(the digits' share, where they are used, is a fourteenth of that and one rounding), one per
chunk of 128, one for alpha, one for beta C: (1.1 K + 4) 2^-53 (|alpha| t + |beta C|), and
half a subnormal for each product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _check(ctx, a, b, ta="N", tb="N", alpha=1.0, beta=0.0, C0=None):
    k = a.shape[1]
    C0 = np.zeros((a.shape[0], b.shape[1])) if C0 is None else C0
    out = ctx.dgemm(a.T.copy() if ta == "T" else a, b.T.copy() if tb == "T" else b, ta, tb, alpha, beta, C=C0)
    x, y = a.astype(LD), b.astype(LD)
    ref = alpha * (x @ y) + beta * C0.astype(LD)
    t = abs(alpha) * (np.abs(x) @ np.abs(y)) + abs(beta) * np.abs(C0.astype(LD))
    tol = (1.1 * k + 4) * LD(2.0) ** -53 * t + k * LD(2.0) ** -1074
    err = np.abs(out.astype(LD) - ref)
    assert (err <= tol).all(), float((err / np.maximum(tol, LD(5e-324))).max())


def test_one_small_element(ctx):
    _check(ctx, np.array([[1.0, 1e-20]]), np.array([[0.0], [1.0]]))
    _check(ctx, np.diag(10.0 ** np.arange(-30.0, 30.0)), np.ones((60, 3)))


def test_falling_row_against_rising_column(ctx):
    r = 10.0 ** np.linspace(0, -20, 64)
    rng = np.random.default_rng(2)
    _check(ctx, r[None] * rng.uniform(0.5, 1.5, (40, 64)), r[::-1, None] * rng.uniform(0.5, 1.5, (64, 40)))


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (7, 9, 15), (31, 33, 17), (33, 31, 129), (64, 65, 127), (130, 7, 257)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
def test_sparse_and_graded(ctx, m, n, k, ta, tb):
    rng = np.random.default_rng(m + 7 * n + 31 * k)
    for decades in (3, 12, 40):
        a = rng.standard_normal((m, k)) * 10.0 ** rng.uniform(-decades, decades, (m, k)) * (rng.random((m, k)) < 0.3)
        b = rng.standard_normal((k, n)) * 10.0 ** rng.uniform(-decades, decades, (k, n)) * (rng.random((k, n)) < 0.3)
        alpha, beta = (1.0, 0.0) if m % 2 else (-0.5, 2.0)
        _check(ctx, a, b, ta, tb, alpha, beta, rng.standard_normal((m, n)))


def test_subnormals(ctx):
    rng = np.random.default_rng(4)
    a = rng.standard_normal((35, 20)) * 1e-310
    a[::3] = rng.standard_normal((12, 20))
    a[::3, ::2] *= 1e-312
    _check(ctx, a, rng.standard_normal((20, 37)) * 1e3)
