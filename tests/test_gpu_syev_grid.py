"""The grid-wide FP64 Jacobi (orders above 110: the clean-up behind the FP32 start
vectors up to 512, the whole solve above): every CTA derives each round's rotations
from the same matrix, so repeated solves agree to the last bit.

Residual and orthogonality as for the one-CTA solver: the stopping rule of 1e-14 ||A||_F
and the rounding of the rotations, 1e-13 ||A||_F and 1e-13 sqrt(n)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,repeats", [(111, 12), (224, 12), (301, 12), (513, 3), (644, 3)])
@pytest.mark.parametrize("kind", ["spread", "dense"])
def test_repeated_solves(ctx, n, repeats, kind):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    w = np.linspace(-20.0, 2.0, n) if kind == "spread" else -20.0 + 1e-4 * np.arange(n)
    A = (Q * w) @ Q.T
    A = 0.5 * (A + A.T)
    first = None
    for _ in range(repeats):
        e, V = ctx.syev_batched(A[None].copy())
        e, V = e[0], V[0]
        if first is None:
            first = e, V
            assert np.all(np.diff(e) >= 0)
            assert np.abs(A @ V - V * e).max() < 1e-13 * np.linalg.norm(A)
            assert np.abs(V.T @ V - np.eye(n)).max() < 1e-13 * np.sqrt(n)
        assert np.array_equal(e, first[0]) and np.array_equal(V, first[1])
