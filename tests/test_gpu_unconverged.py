"""What an SCF that runs out of iterations leaves in its outputs."""
import ctypes

import numpy as np
import pytest

from hfsolver_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tolP", [(5, 1e-9), (12, 1e-9), (12, 1e-12)])
@pytest.mark.parametrize("nscf", [1, 2, 5])
@pytest.mark.parametrize("alpha", [1.0, 0.4])
def test_doscf_returns_the_mixed_density(n, tolP, nscf, alpha):
    """Without two-electron integrals every iteration's own density is twice the projector D
    on the lowest states of H, and mixing from 0 leaves (1 - (1 - alpha)^nscf) D.  Spectrum
    within 8 of a gap of 1: 1e-13 times that, and n of roundoff."""
    rng = np.random.default_rng(n)
    nocc = n // 3
    lam = np.sort(np.concatenate([rng.uniform(-4.0, -0.5, nocc), rng.uniform(0.5, 4.0, n - nocc)]))
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    H = np.asfortranarray((Q * lam) @ Q.T)
    m = n * (n + 1) // 2
    int2, S = np.zeros(m * (m + 1) // 2), np.eye(n)
    C, P, w, E0, it = np.zeros((n, n), order="F"), np.zeros((n, n), order="F"), np.zeros(n), np.zeros(1), ctypes.c_int()
    d = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    rc = _lib.lib().hfgpu_doscf(n, d(H), d(int2), d(S), nocc, nscf, 0.0, tolP, alpha, d(C), d(P), d(w), d(E0),
                                ctypes.byref(it))
    assert rc == _lib.ERR_NOT_CONVERGED
    D = 2.0 * Q[:, :nocc] @ Q[:, :nocc].T
    assert np.max(np.abs(P - (1.0 - (1.0 - alpha) ** nscf) * D)) < 8e-13 + n * 1e-15
    assert np.max(np.abs(np.abs(C.T @ Q) - np.eye(n))) < 8e-13 + n * 1e-15 and np.max(np.abs(w - lam)) < 1e-12
