"""G(x) and G(K : x) on grids whose transforms use every radix of the shared-memory passes
(3, 5, 6, 7, 9, 11, 13, primes above 13 and their products), against numpy's FFT in FP64."""
import numpy as np
import pytest

from cpfft_gb300 import rve


def green_ref(x, N, centered):
    f = np.arange(N)
    if centered:
        q1 = np.where(f <= (N - 1) // 2, f, f - N).astype(float)
    else:
        half = (N + 1) // 2 if N % 2 else N // 2 + 1
        q1 = ((f - half) % N + 1 - half).astype(float)
    q = np.stack(np.meshgrid(q1, q1, q1, indexing="ij"))
    qq = (q * q).sum(0)
    inv = np.where(qq > 0, 1.0 / np.where(qq > 0, qq, 1.0), 0.0)
    if centered and N % 2 == 0:
        inv[N // 2], inv[:, N // 2], inv[:, :, N // 2] = 0.0, 0.0, 0.0
    X = np.fft.fftn(x.reshape(3, 3, N, N, N), axes=(2, 3, 4))
    Y = ((X * q).sum(1) * inv)[:, None] * q[None]
    return np.fft.ifftn(Y, axes=(2, 3, 4)).real.reshape(9, N ** 3)


# first stages of 2..13, a prime above 13 alone and with 2 and 3, squares, 2- and 3-stage
# plans on both sides of every rule (split stages 16, three passes 48 and 80, blocks 20, 36, 44)
SIZES = [2, 3, 6, 7, 9, 11, 13, 16, 17, 18, 19, 22, 26, 33, 34, 35, 36, 39, 43, 45, 48, 49, 51, 61,
         63, 66, 80, 81]


@pytest.mark.gpu
@pytest.mark.parametrize("N", SIZES)
def test_green_every_radix(gpulib, N):
    # a transform accumulates at most sum(radices) <= N rounded terms per value and axis, six
    # of them (three axes, there and back): 8 N units of round-off in the 2-norm
    rng = np.random.default_rng(N)
    K = rng.standard_normal((81, N ** 3))
    x = rng.standard_normal((9, N ** 3))
    Kx = (K.reshape(9, 9, -1) * x).sum(1)
    one = np.ones(N ** 3, dtype=np.int32)
    for centered in (False, True):
        s = gpulib.Solver(N, one, np.zeros((3, N ** 3)), [dict(rve.FCC_VOCE)], 1.0,
                          gpulib.G_CENTERED if centered else gpulib.G_REF_SHIFT)
        try:
            s.set_K4(K)
            # the contraction K : x cancels in part: its error is relative to |K| |x|
            big = np.linalg.norm((np.abs(K).reshape(9, 9, -1) * np.abs(x)).sum(1))
            for flgK, src, scale in ((False, x, np.linalg.norm(x)), (True, Kx, big)):
                ref = green_ref(src, N, centered)
                y = s.G_K_dF(x, flgK)
                assert np.linalg.norm(y - ref) <= 8 * N * 2.0 ** -53 * scale
            s.set_mode(gpulib.PREC_MIXED)
            ref = green_ref(x, N, centered)
            y = s.G_K_dF_f32(x.astype(np.float32), False)
            assert np.linalg.norm(y - ref) <= 8 * N * 2.0 ** -24 * np.linalg.norm(x)
        finally:
            s.close()
