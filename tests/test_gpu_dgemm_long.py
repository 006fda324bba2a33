"""mq_dgemm with few elements and a long K, which is split over the SMs: both sides of
the line (three chunks of 128), parts of one and of several chunks, a ragged last chunk,
alpha and beta, each transposition, both operands as the one with more tiles.

Bound per element as for any FP64 sum in chunks of 128 (at most 128 roundings inside one,
then one per chunk and part, alpha and beta): (140 + 2 K/128) 2^-53 (|alpha| sum |a||b| + |beta C|)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.mark.parametrize("m,n,k", [(32, 32, 384), (32, 32, 385), (1, 1, 512), (33, 7, 1000), (5, 300, 2049),
                                   (200, 200, 1537), (32, 32, 20001)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
def test_long_k(ctx, m, n, k, ta, tb):
    rng = np.random.default_rng(m + 7 * n + 31 * k)
    a, b, C0 = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    alpha, beta = (1.0, 0.0) if n % 2 else (-0.5, 2.0)
    out = ctx.dgemm(a.T.copy() if ta == "T" else a, b.T.copy() if tb == "T" else b, ta, tb, alpha, beta, C=C0)
    cols = rng.permutation(n)[:8]  # (extended precision is slow)
    x, y, z = a.astype(LD), b[:, cols].astype(LD), C0[:, cols].astype(LD)
    t = abs(alpha) * (np.abs(x) @ np.abs(y)) + abs(beta) * np.abs(z)
    err = np.abs(out[:, cols].astype(LD) - (alpha * (x @ y) + beta * z))
    assert (err <= (140 + 2 * k / 128) * LD(2.0) ** -53 * t).all()
