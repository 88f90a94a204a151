"""The FP64 CG of small grids (one launch, split or butterfly stages) and of the first grid
above them: the true residual of the returned x, in FP64 with numpy's FFT."""
import numpy as np
import pytest

from cpfft_gb300 import rve
from test_green_radices import green_ref


@pytest.mark.gpu
@pytest.mark.parametrize("N,centered", [(2, True), (3, False), (5, False), (8, True), (11, False),
                                        (12, True), (13, False), (16, True), (17, False),
                                        (32, True), (33, False), (34, True)])
def test_cg_small_grids(gpulib, N, centered):
    rng = np.random.default_rng(N)
    # a symmetric positive definite tangent per voxel, condition number about 20
    A = rng.standard_normal((N ** 3, 9, 9)) * 0.4
    K = np.einsum("vij,vkj->vik", A, A) + np.eye(9)
    K4 = np.ascontiguousarray(K.reshape(N ** 3, 81).T)

    def op(x):
        return green_ref((K4.reshape(9, 9, -1) * x).sum(1), N, centered)

    b = op(rng.standard_normal((9, N ** 3)))
    one = np.ones(N ** 3, dtype=np.int32)
    s = gpulib.Solver(N, one, np.zeros((3, N ** 3)), [dict(rve.FCC_VOCE)], 1.0,
                      gpulib.G_CENTERED if centered else gpulib.G_REF_SHIFT)
    try:
        s.set_K4(K4)
        tol = 1e-8
        x, its = s.fftPcg(b, tol)
        x2, its2 = s.fftPcg(b, tol)
        assert its == its2 and np.array_equal(x, x2)  # fixed-order sums: runs repeat exactly
        # stops at tol ||b|| (or tol) on the recursion's residual, which round-off moves from
        # the true one by a few units per iteration: far below 1 % of 1e-8
        limit = max(tol * np.linalg.norm(b), tol)
        assert np.linalg.norm(b - op(x)) <= 1.01 * limit
        assert np.isfinite(x).all() and (its >= 1 or np.linalg.norm(b) < 1e-15)
        # a zero right-hand side returns at once
        x0, it0 = s.fftPcg(np.zeros_like(b), tol)
        assert it0 == 0 and not x0.any()
        # a non-finite one is an error, and the context stays usable
        bad = b.copy()
        bad[0, 0] = np.inf
        with pytest.raises(gpulib.CpfftError) as e:
            s.fftPcg(bad, tol)
        assert e.value.code == -10
        assert np.array_equal(s.fftPcg(b, tol)[0], x)
    finally:
        s.close()
