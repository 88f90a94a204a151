"""The two-voxels-a-warp local solve of the dislocation-density laws where its tiling can go
wrong: grids whose voxel count leaves a partial block or a partial warp, voxels of another
material between crystals, unloaded voxels beside loaded ones, explicit and implicit passes and
a second step, against the oracle."""
import numpy as np
import pytest

from cpfft_gb300 import rve


def per_voxel(a, b):
    scale = np.maximum(np.abs(b).max(axis=0), 1e-6 * np.abs(b).max())
    return (np.abs(a - b).max(axis=0) / scale).max()


@pytest.mark.gpu
@pytest.mark.parametrize("law", ["mrr", "ornl"])
@pytest.mark.parametrize("N,mixed,idle", [(2, False, False), (3, False, True), (3, True, False),
                                          (5, True, True), (6, False, True)])
def test_mrr_partial_groups(gpulib, oracle, law, N, mixed, idle):
    crystal = rve.MRR_FCC if law == "mrr" else rve.ORNL_FCC
    r = rve.make_rve(N, 3, 17 + N, crystal)
    mats = np.array(r.mat_list)
    crystals = list(r.crystals)
    N3 = N ** 3
    if mixed:
        crystals.append(rve.NOT_A_CRYSTAL)
        mats[np.arange(N3) % 3 == 1] = 2
    s = gpulib.Solver(N, mats, r.kocks, crystals, 1.0, gpulib.G_REF_SHIFT)
    o = oracle.Oracle(N, mats, r.kocks, crystals, 1.0, 0, nthreads=4)
    try:
        if mixed:
            s.set_mises(2, **rve.MM01_DECK[0])
            o.set_mises(2, rve.MM01_DECK[0])
        rng = np.random.default_rng(5)
        F0 = np.zeros((9, N3))
        F0[[0, 4, 8]] = 1.0
        d1 = 1e-3 * rng.standard_normal((9, N3))
        d2 = 1e-3 * rng.standard_normal((9, N3))
        if idle:  # no load in the first step: mm10's early return, an explicit state
            d1[:, np.arange(N3) % 4 == 2] = 0.0
        F1 = F0 + d1
        F2 = F1 + d2
        for step, it, Fa, Fb in ((1, 0, F0, F1), (1, 1, F0, F1), (2, 0, F1, F2), (2, 2, F1, F2)):
            P, K, rc = s.drive_eps_sig(step, it, Fa, Fb, want_K4=True)
            Po, Ko, fails, _ = o.stress_update(step, it, Fa, Fb)
            assert rc == (1 if fails else 0)
            # the bounds of the laws' parity test (tests/test_mrr.py)
            assert per_voxel(P, Po) < 1e-8
            assert per_voxel(K, Ko) < 1e-7
            if step == 1 and it == 1:
                s.commit()
                o.commit()
    finally:
        s.close()
        o.close()
