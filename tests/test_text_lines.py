"""Element lines where the 32-voxel blocks of the formatter can go wrong: a partial last block,
a partial last 16 bytes, values the device leaves to the host among others, both quantities;
against the oracle's restatement."""
import numpy as np
import pytest

from cpfft_gb300 import rve


@pytest.mark.gpu
@pytest.mark.parametrize("N,scale", [(2, 1e-3), (3, 1e-3), (5, 1e-22), (7, 1e-3), (8, 3e-18)])
def test_format_flat_blocks(gpulib, N, scale):
    from oracle import flat_ref
    r = rve.make_rve(N, 2, 9)
    s = gpulib.Solver(N, r.mat_list, r.kocks, r.crystals, 1.0, gpulib.G_REF_SHIFT)
    try:
        rng = np.random.default_rng(N)
        F0 = np.zeros((9, N ** 3))
        F0[[0, 4, 8]] = 1.0
        s.drive_eps_sig(1, 1, F0, F0 + scale * rng.standard_normal((9, N ** 3)))
        s.commit()
        H = s.fields(history=True)[2]
        for quantity, word, nvals in ((2, 0, 26), (1, 23, 22)):
            got = s.format_flat(quantity)
            assert got == flat_ref.flat_text(H[word:word + 6], nvals).encode()
            assert s.format_flat(quantity) == got
    finally:
        s.close()
