"""The one-CTA eigensolver on dense spectra: many levels 1e-5 to 2e-3 of the norm apart,
whose first-order rotations are small each and large together, from FP32 start vectors.

A cold FP64 Jacobi makes some three sweeps of n - 1 rotations of every column, each
rounded twice: 6 n 2^-53 in a column's norm if all had the same sign, 7e-14 at n = 110.
So 1e-13 for V^T V - I, and the same of the norm for the eigenvalues and the residual."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 33, 56, 64, 65, 80, 81, 110])
@pytest.mark.parametrize("spacing", [1e-5, 3e-5, 1e-4, 2e-4, 5e-4, 2e-3])
def test_syev_dense_spectrum(ctx, n, spacing):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * (-20.0 + 20.0 * spacing * np.arange(n))) @ Q.T
    A = 0.5 * (A + A.T)
    w, V = ctx.syev_batched(A[None].copy())
    w, V = w[0], V[0]
    norm = np.linalg.norm(A, 2)
    assert np.abs(V.T @ V - np.eye(n)).max() < 1e-13
    assert np.abs(w - np.linalg.eigvalsh(A)).max() < 1e-13 * norm
    assert np.abs(A @ V - V * w).max() < 1e-13 * norm
