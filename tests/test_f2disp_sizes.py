"""Nodal displacements at the sizes where the folded transforms can go wrong: odd and even N
(the middle point), line counts that leave a partial tile of 32, the smallest grids, unequal
box sides; against the oracle's element assembly."""
import numpy as np
import pytest

from cpfft_gb300 import rve


@pytest.mark.gpu
@pytest.mark.parametrize("N,lengths", [(2, (1.0, 1.0, 1.0)), (3, (100.0, 50.0, 20.0)),
                                       (4, (1.0, 2.0, 3.0)), (5, (7.0, 7.0, 7.0)),
                                       (10, (100.0, 10.0, 30.0))])
def test_f2disp_sizes(gpulib, N, lengths):
    from oracle import f2disp_ref
    rng = np.random.default_rng(N)
    F = np.zeros((9, N ** 3))
    F[[0, 4, 8]] = 1.0
    F += 0.02 * rng.standard_normal(F.shape)
    s = gpulib.Solver(N, np.ones(N ** 3, np.int32), np.zeros((3, N ** 3)), [dict(rve.FCC_VOCE)], 1.0,
                      gpulib.G_REF_SHIFT)
    try:
        s.set_F(None, F)
        u = s.f2disp(lengths)
        ref = f2disp_ref.displacements(F, N, lengths)
        # the bound of tests/test_f2disp.py: 1e-12 of the box
        assert np.abs(u - ref).max() < 1e-12 * max(lengths) * 10
        assert np.array_equal(u, s.f2disp(lengths))
    finally:
        s.close()
