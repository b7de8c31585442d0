"""Densities of the SCF by purification on constant Fock matrices of chosen spectra: with
no two-electron integrals every iteration sees the same F, so the second one knows its
gap and steps stretched."""
import numpy as np
import pytest

import hfsolver_gb300 as hf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nocc,gap", [(7, 3, 0.5), (8, 1, 0.5), (8, 7, 1e-2), (9, 4, 0.0), (17, 8, 1e-5), (40, 11, 0.3),
                                        (65, 30, 1e-3)])
def test_doscf_of_a_fixed_spectrum(n, nocc, gap):
    """P is twice the projector on the lowest nocc states and E0 their sum, through a gap
    that is wide, narrow (more steps than are kept on record) or none (an eigensolve).
    Spectrum within [-20, 4]; sums of n terms of unit roundoff 1.1e-16 and condition
    |lambda| / gap of the projector: 1e-11 on E0, and on P 1e-13 * 24 / gap."""
    rng = np.random.default_rng(7 * n + nocc)
    lam = np.sort(np.concatenate([rng.uniform(-20.0, -1.0, nocc), rng.uniform(1.0, 4.0, n - nocc)]))
    lam[nocc - 1] = -0.4
    lam[nocc] = lam[nocc - 1] + gap
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    H = (Q * lam) @ Q.T
    H = 0.5 * (H + H.T)
    m = n * (n + 1) // 2
    L = np.eye(n) + 0.1 / np.sqrt(n) * np.tril(rng.standard_normal((n, n)), -1)  # S = L L^T is near I
    r = hf.doscf(L @ H @ L.T, np.zeros(m * (m + 1) // 2), L @ L.T, nocc, 20, 1e-9, 1e-8, 1.0)
    C, P, w, E0 = r[0], r[1], r[2], r[3]
    assert abs(E0 - 2.0 * lam[:nocc].sum()) < 1e-11 * max(1.0, abs(lam).sum())
    assert np.abs(w - lam).max() < 1e-11
    if gap > 0:
        D = 2.0 * Q[:, :nocc] @ Q[:, :nocc].T
        got = L.T @ P @ L
        assert np.abs(got - D).max() < 1e-13 * 24.0 / gap
