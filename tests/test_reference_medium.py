"""Ellipticity of the preconditioner's reference medium (krylov.cu, k_medium) against NumPy:
the least det A / tr(A)^3 of the acoustic tensor over 65 x 128 directions, its acceptance
threshold of 1e-9 from both sides, and the refusal of a medium that is not elliptic."""
import re

import numpy as np
import pytest

from cpfft_gb300 import rve

pytestmark = pytest.mark.gpu


def _diag(first):
    K = np.eye(9)
    K[:3, :3] *= first
    return K


def _isotropic():
    d = np.eye(3)
    return (1.2e5 * np.einsum("ij,kl->ijkl", d, d) + 8.0e4 * (np.einsum("ik,jl->ijkl", d, d)
            + np.einsum("il,jk->ijkl", d, d))).reshape(9, 9)


def _random():
    A = np.random.default_rng(3).standard_normal((9, 9))
    return A @ A.T + 0.5 * np.random.default_rng(4).standard_normal((9, 9))


MEDIA = {"isotropic": _isotropic(), "random": _random(), "above": _diag(8.1e-9),
         "below": _diag(7.9e-9), "indefinite": _diag(-1.0)}


def _least(K):
    K = K.astype(np.float32).astype(np.float64)
    K = (0.5 * (K + K.T)).reshape(3, 3, 3, 3)
    th = np.pi * np.arange(65)[:, None] / 64
    ph = 2 * np.pi * np.arange(128)[None] / 128
    n = np.stack(np.broadcast_arrays(np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)))
    A = np.einsum("ijkl,jab,lab->abik", K, n, n)
    if np.linalg.eigvalsh(A).min() <= 0:
        return None
    return (np.linalg.det(A) / np.trace(A, axis1=2, axis2=3) ** 3).min()


@pytest.mark.parametrize("name", sorted(MEDIA))
def test_ellipticity(gpulib, name, monkeypatch, capfd):
    N, K = 9, MEDIA[name]
    monkeypatch.setenv("CPFFT_LOG", "1")
    s = gpulib.Solver(N, np.ones(N ** 3, np.int32), np.zeros((3, N ** 3)), [dict(rve.FCC_VOCE)], 1.0,
                  gpulib.G_CENTERED)
    s.set_mode(gpulib.PREC_MIXED, 0)
    s.set_precond(gpulib.PRECOND_REFERENCE)
    capfd.readouterr()
    s.set_K4(np.repeat(K.reshape(81, 1), N ** 3, axis=1))
    s.close()
    line = re.search(r"acoustic tensor (\S+)( \(not used\))?", capfd.readouterr().err)
    want = _least(K)
    if want is None:
        assert line is None
    else:  # the line has four digits: half a unit of the last is at most 5e-4
        assert abs(float(line.group(1)) / want - 1) < 5.1e-4
        assert (line.group(2) is None) == (want > 1e-9)
