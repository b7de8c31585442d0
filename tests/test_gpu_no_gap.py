"""SCF iterations of systems without a gap: a purification that finds none is not repeated
every iteration."""
import numpy as np
import pytest

import hfsolver_gb300 as hf
from hfsolver_gb300 import _lib

pytestmark = pytest.mark.gpu


def _system(n, nocc, gap, coupling):
    rng = np.random.default_rng(n)
    lam = np.sort(np.concatenate([rng.uniform(-20.0, -1.0, nocc), rng.uniform(1.0, 4.0, n - nocc)]))
    lam[nocc - 1] = -0.4
    lam[nocc] = lam[nocc - 1] + gap
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    H = (Q * lam) @ Q.T
    m = n * (n + 1) // 2
    B = rng.standard_normal((m, 3))
    k, l = np.tril_indices(m)
    return 0.5 * (H + H.T), coupling * np.einsum("ik,ik->i", B[k], B[l])


def _launches(n, nocc, H, int2, nscf, tolP):
    """Kernels of nscf iterations that cannot converge; tolP < 1e-11 solves for the
    eigenvectors every time."""
    L = _lib.lib()
    k0 = L.hfgpu_kernel_launches()
    with pytest.raises(hf.SCFNotConverged):
        hf.doscf(H, int2, np.eye(n), nocc, nscf, 0.0, tolP, 1.0)
    return L.hfgpu_kernel_launches() - k0


@pytest.mark.parametrize("n,gap", [(9, 0.0), (25, 0.0), (25, 1e-6), (60, 1e-12)])
def test_one_failed_purification_at_most(n, gap):
    """Beyond the eigensolves' kernels no more than one purification's (five and the
    report's) in 20 iterations of the same F."""
    H, int2 = _system(n, n // 3, gap, 0.0)
    assert _launches(n, n // 3, H, int2, 20, 1e-9) <= _launches(n, n // 3, H, int2, 20, 1e-12) + 6


def test_purification_returns_with_the_gap():
    """The core Hamiltonian has no gap, the Fock matrices after it do: from the third
    iteration on the density comes from a purification, with fewer kernels."""
    n, nocc = 24, 8
    H, int2 = _system(n, nocc, 0.0, 0.02)
    eig, sp2 = _launches(n, nocc, H, int2, 20, 1e-12), _launches(n, nocc, H, int2, 20, 1e-9)
    alone = _launches(n, nocc, *_system(n, nocc, 0.0, 0.0), 20, 1e-9)
    assert sp2 <= eig - 3 * 16 and alone > eig - 3


def test_one_narrow_gap_costs_no_eigensolve():
    """A first Fock matrix with a gap of 1e-4 (70 steps) and wide ones after it take the same
    kernels as wide ones throughout."""
    n, nocc = 24, 8
    k = [_launches(n, nocc, *_system(n, nocc, gap, 0.02), 12, 1e-9) for gap in (1e-4, 0.5)]
    assert k[0] == k[1]
