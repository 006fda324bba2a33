"""FP64 products from fixed-point digits on the tensor cores (mq_dgemm) against
extended precision, at the edges of their tiles (32, 64), fragments (8, 16) and
K chunks (128), for every transposition, alpha and beta, rows of very different
size, and non-finite elements.

Bound per element: one rounding of each K chunk's sum and of the sums between
chunks, 2^-52 of the chunks' absolute sums, plus what the digits leave out: the
operands' rounding and the dropped levels, at most K 2^-59 2^(ea + eb) with
2^ea, 2^eb up to twice the largest element of the row and the column, so K 2^-57
times the product of the two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _bound(a, b):
    k = a.shape[1]
    part = sum(np.abs(a[:, s:s + 128].astype(LD) @ b[s:s + 128].astype(LD)) for s in range(0, k, 128))
    return 2.0 ** -52 * part + k * 2.0 ** -57 * np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :]


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (7, 9, 15), (16, 8, 16), (17, 33, 31), (32, 32, 128), (33, 31, 129),
                                   (64, 65, 127), (130, 7, 257), (1100, 96, 40), (900, 1100, 65)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
def test_dgemm_correct_to_rounding(ctx, m, n, k, ta, tb):
    rng = np.random.default_rng(m + 7 * n + 31 * k)
    a = rng.standard_normal((m, k)) * np.exp(rng.uniform(-25, 25, (m, 1)))  # rows of any size
    b = rng.standard_normal((k, n)) * np.exp(rng.uniform(-8, 8, (k, n)))    # elements of any size
    alpha, beta = (1.0, 0.0) if m % 2 else (-0.5, 2.0)
    C0 = rng.standard_normal((m, n))
    out = ctx.dgemm(a.T.copy() if ta == "T" else a, b.T.copy() if tb == "T" else b, ta, tb, alpha, beta, C=C0)
    ref = (alpha * (a.astype(LD) @ b.astype(LD)) + beta * C0)
    tol = abs(alpha) * _bound(a, b) + 2.0 ** -52 * (np.abs(ref) + abs(beta) * np.abs(C0)) + 1e-300
    assert (np.abs(out - ref) <= tol).all(), float((np.abs(out - ref) / tol).max())


def test_dgemm_non_finite(ctx):
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal((70, 40)), rng.standard_normal((40, 70))
    a[3, 7], a[50, 1], b[11, 66] = np.inf, np.nan, -np.inf
    out = ctx.dgemm(a, b)
    with np.errstate(invalid="ignore"):
        ref = a @ b
    assert np.array_equal(np.isnan(out), np.isnan(ref)) and np.array_equal(np.isposinf(out), np.isposinf(ref))
    fin = np.isfinite(ref)
    assert np.abs(out[fin] - ref[fin]).max() < 1e-13
