"""J - K/2 from the packed array against the definition, index by index."""
import numpy as np
import pytest

import hfsolver_gb300 as hf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 9, 33])
def test_formG_from_random_packed_integrals(n):
    """G_ij = sum_kl P_kl [(ij|kl) - (il|kj)/2] with the integrals unpacked: sums of n^2
    terms of magnitude below 20 (normal deviates), 1.5 n^2 20 1.1e-16 on both sides."""
    rng = np.random.default_rng(n)
    m = n * (n + 1) // 2
    ints = rng.standard_normal(m * (m + 1) // 2)
    ints[rng.random(ints.size) < 0.2] = 0.0  # as a screened array has
    P = rng.standard_normal((n, n))
    P = P + P.T
    i = np.arange(n)
    hi, lo = np.maximum(i[:, None], i[None, :]), np.minimum(i[:, None], i[None, :])
    pair = hi * (hi + 1) // 2 + lo
    M = np.zeros((m, m))
    M[np.tril_indices(m)] = ints
    M += np.tril(M, -1).T
    V = M[pair][:, :, pair]  # (ij|kl)
    want = np.einsum("ijkl,kl->ij", V, P) - 0.5 * np.einsum("ilkj,kl->ij", V, P)
    assert np.abs(hf.formG(P, ints) - want).max() < 1.5 * n * n * 20 * 2.2e-16 + 1e-15
