"""The stress update for rate exponents on every branch of the power: integral ones (binary
powering), non-integral ones up to 9 (the exponent's table) and above (pow), against the oracle
over two steps, for 12 systems and 48."""
import numpy as np
import pytest

from cpfft_gb300 import rve


@pytest.mark.gpu
@pytest.mark.parametrize("base,n", [("fcc", 2.0), ("fcc", 2.5), ("fcc", 8.75), ("fcc", 9.0),
                                    ("fcc", 9.5), ("fcc", 20.0), ("bcc48", 3.25), ("bcc48", 10.5)])
def test_stress_update_rate_exponents(gpulib, oracle, base, n):
    N = 5
    crystal = dict(rve.FCC_VOCE if base == "fcc" else rve.BCC48_DECK, harden_n=n, exact_j22=1)
    dt = 1.0 if base == "fcc" else 10.0
    r = rve.make_rve(N, 4, 71, crystal)
    s = gpulib.Solver(N, r.mat_list, r.kocks, r.crystals, dt, gpulib.G_REF_SHIFT)
    o = oracle.Oracle(N, r.mat_list, r.kocks, r.crystals, dt, 0, nthreads=8)
    try:
        rng = np.random.default_rng(3)
        F0 = np.zeros((9, N ** 3))
        F0[[0, 4, 8]] = 1.0
        F1 = F0 + 2e-3 * rng.standard_normal((9, N ** 3))
        F2 = F1 + 2e-3 * rng.standard_normal((9, N ** 3))
        for step, Fa, Fb in ((1, F0, F1), (2, F1, F2)):
            P, K, rc = s.drive_eps_sig(step, 1, Fa, Fb, want_K4=True)
            Po, Ko, fails, _ = o.stress_update(step, 1, Fa, Fb)
            assert rc == (1 if fails else 0)
            # both solve the local equations to 1e-10 of their first residual: the bounds of the
            # other parity tests of P (1e-8) and, with the amplified tangent, of dP/dF (5e-7)
            assert np.abs(P - Po).max() < 1e-8 * np.abs(Po).max()
            assert np.abs(K - Ko).max() < 5e-7 * np.abs(Ko).max()
            s.commit()
            o.commit()
    finally:
        s.close()
        o.close()
