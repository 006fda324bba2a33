"""The one-CTA eigensolver (orders up to 110) against its defining equations:
A V = V diag(w), V^T V = I, w ascending, at the smallest orders, at odd and
even ones, at both sides of the order where its scratch leaves shared memory
(80), and at its largest; for well separated, clustered and repeated
eigenvalues and for matrices far from unit scale.

Tolerance: the solver stops at ||offdiag||_F <= 1e-14 ||A||_F; the rotations
and products add rounding of a few n eps, so 1e-13 ||A||_F bounds the residual
at these orders with a margin of about five, and 1e-13 sqrt(n) the
orthogonality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, kind, rng):
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    if kind == "spread":
        w = np.linspace(-20.0, 2.0, n)
    elif kind == "clusters":  # levels 1e-9 apart, as core levels of a cluster of molecules
        w = np.where(np.arange(n) < n // 2, -20.0 + 1e-9 * np.arange(n), 0.1 * np.arange(n))
    elif kind == "repeated":
        w = np.repeat([-1.0, 3.0], [n // 2, n - n // 2]).astype(float)
    else:
        w = rng.standard_normal(n) * float(kind)
    A = (Q * w) @ Q.T
    return 0.5 * (A + A.T)


@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 33, 56, 80, 81, 110])
@pytest.mark.parametrize("kind", ["spread", "clusters", "repeated", "1e-200", "1e120"])
def test_syev_one_cta(ctx, n, kind):
    rng = np.random.default_rng(n)
    A = np.stack([_matrix(n, kind, rng) for _ in range(2)])
    w, V = ctx.syev_batched(A.copy())
    for a, e, v in zip(A, w, V):
        big = max(np.abs(a).max(), 1e-300)  # (an order-1 cluster is the zero matrix)
        scale = np.sqrt(np.sum((a / big) ** 2)) * big + (big == 1e-300)
        assert np.all(np.diff(e) >= 0)
        r = np.abs(a / scale @ v - v * (e / scale)).max()
        assert r < 1e-13, (n, kind, r)
        assert np.abs(v.T @ v - np.eye(n)).max() < 1e-13 * np.sqrt(n), (n, kind)


def test_syev_diagonal_and_zero(ctx):
    A = np.stack([np.zeros((7, 7)), np.diag(np.arange(7.0)[::-1])])
    w, V = ctx.syev_batched(A.copy())
    assert np.array_equal(w[0], np.zeros(7)) and np.allclose(w[1], np.arange(7.0), atol=1e-15)
    for v in V:
        assert np.abs(v.T @ v - np.eye(7)).max() < 1e-14
