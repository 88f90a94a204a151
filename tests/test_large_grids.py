"""Grids of the shared-memory passes above 81 points a side, up to the largest that cpfft_init
takes: their contexts exist in both precisions, and G(x) (with G(K : x) on the smaller ones)
agrees with numpy's FFT in FP64."""
import numpy as np
import pytest

from cpfft_gb300 import rve
from test_green_radices import green_ref


# 111 and 112: a plane of the three-pass form fits a block's shared memory, and no longer does;
# 125 = 5^3; 127 and 251 primes (251: the largest); 160 = 2^5 5; 255 = 3 5 17
@pytest.mark.gpu
@pytest.mark.parametrize("N,centered", [(111, True), (112, False), (125, False), (127, True),
                                        (160, True), (251, False), (255, True)])
def test_green_large_grids(gpulib, N, centered):
    rng = np.random.default_rng(N)
    x = rng.standard_normal((9, N ** 3))
    one = np.ones(N ** 3, dtype=np.int32)
    s = gpulib.Solver(N, one, np.zeros((3, N ** 3)), [dict(rve.FCC_VOCE)], 1.0,
                      gpulib.G_CENTERED if centered else gpulib.G_REF_SHIFT)
    try:
        # the bound of test_green_radices.py: 8 N units of round-off in the 2-norm
        ref = green_ref(x, N, centered)
        assert np.linalg.norm(s.G_K_dF(x, False) - ref) <= 8 * N * 2.0 ** -53 * np.linalg.norm(x)
        if N <= 127:
            K = rng.standard_normal((81, N ** 3))
            s.set_K4(K)
            Kx = (K.reshape(9, 9, -1) * x).sum(1)
            big = np.linalg.norm((np.abs(K).reshape(9, 9, -1) * np.abs(x)).sum(1))
            err = np.linalg.norm(s.G_K_dF(x, True) - green_ref(Kx, N, centered))
            assert err <= 8 * N * 2.0 ** -53 * big
        s.set_mode(gpulib.PREC_MIXED)
        y = s.G_K_dF_f32(x.astype(np.float32), False)
        assert np.linalg.norm(y - ref) <= 8 * N * 2.0 ** -24 * np.linalg.norm(x)
    finally:
        s.close()
