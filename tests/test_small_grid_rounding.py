"""Rounding of the operator on grids of up to 16 points (split transform stages): no further from
long double than the five-pass operator with register butterflies and direct sums."""
import numpy as np
import pytest

from cpfft_gb300 import rve

# the five-pass operator's distance from long double on the fields below: mean of the relative
# 2-norms, 1e-16 (it has no split stages).  The mean of twelve fields of 9 N^3 values differs by
# 1 / sqrt(2 12 9 N^3), 0.4 % at most, from that of others: 3 % is a change of the rounding.
FIVE_PASS = {7: 3.01, 11: 3.54, 13: 3.69, 16: 3.37}


def green_longdouble(x, N, centered):
    f = np.arange(N)
    if centered:
        q1 = np.where(f <= (N - 1) // 2, f, f - N).astype(np.longdouble)
    else:
        half = (N + 1) // 2 if N % 2 else N // 2 + 1
        q1 = ((f - half) % N + 1 - half).astype(np.longdouble)
    a = 2 * np.longdouble("3.14159265358979323846264338327950288") * (np.outer(f, f) % N) / N
    W = np.cos(a) - 1j * np.sin(a)
    X = x.astype(np.clongdouble).reshape(9, N, N, N)
    for ax in (1, 2, 3):
        X = np.moveaxis(np.tensordot(X, W, axes=([ax], [1])), -1, ax)
    q = np.stack(np.meshgrid(q1, q1, q1, indexing="ij"))
    qq = (q * q).sum(0)
    inv = np.where(qq > 0, 1 / np.where(qq > 0, qq, 1), 0)
    if centered and N % 2 == 0:
        inv[N // 2], inv[:, N // 2], inv[:, :, N // 2] = 0, 0, 0
    Y = ((X.reshape(3, 3, N, N, N) * q).sum(1) * inv)[:, None] * q[None]
    Y = Y.reshape(9, N, N, N)
    for ax in (1, 2, 3):
        Y = np.moveaxis(np.tensordot(Y, W.conj() / N, axes=([ax], [1])), -1, ax)
    return Y.real.reshape(9, -1)


@pytest.mark.gpu
@pytest.mark.parametrize("N", sorted(FIVE_PASS))
def test_small_grid_rounding(gpulib, N):
    err = []
    one = np.ones(N ** 3, dtype=np.int32)
    for centered in (False, True):
        s = gpulib.Solver(N, one, np.zeros((3, N ** 3)), [dict(rve.FCC_VOCE)], 1.0,
                          gpulib.G_CENTERED if centered else gpulib.G_REF_SHIFT)
        try:
            for seed in range(6):
                x = np.random.default_rng(100 * N + seed).standard_normal((9, N ** 3))
                ref = green_longdouble(x, N, centered)
                err.append(float(np.linalg.norm((s.G_K_dF(x, False) - ref).astype(float)) /
                                 np.linalg.norm(ref.astype(float))))
        finally:
            s.close()
    assert np.mean(err) <= 1.03e-16 * FIVE_PASS[N]
