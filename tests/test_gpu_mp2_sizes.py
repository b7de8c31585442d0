"""MBPT2 from packed integrals at sizes on both sides of the row maxima's run lengths (64
and 128 functions) and of the 32-wide tiles of the energy sum."""
import numpy as np
import pytest

import hfsolver_gb300 as hf

pytestmark = pytest.mark.gpu


def _energy(n, o, ints, C, lam):
    """The energy in plain FP64 numpy, from the packed integrals' symmetric pair matrix."""
    i = np.arange(n)
    hi, lo = np.maximum(i[:, None], i[None, :]), np.minimum(i[:, None], i[None, :])
    pair = hi * (hi + 1) // 2 + lo
    m = n * (n + 1) // 2
    M = np.zeros((m, m))
    M[np.tril_indices(m)] = ints
    M += np.tril(M, -1).T
    C1, C2 = C[:, :o], C[:, o:]
    Z = np.empty((m, o, n - o))
    for p0 in range(0, m, 512):
        Z[p0:p0 + 512] = np.einsum("pls,si,la->pia", M[p0:p0 + 512][:, pair], C1, C2, optimize=True)
    X = np.einsum("mnia,mj,nb->iajb", Z[pair], C1, C2, optimize=True)
    d = lam[:o, None, None, None] - lam[None, o:, None, None] + lam[None, None, :o, None] - lam[None, None, None, o:]
    t = X * (2.0 * X - X.transpose(0, 3, 2, 1)) / d
    return t.sum(), np.abs(t).sum()


@pytest.mark.parametrize("n,o", [(9, 2), (64, 31), (65, 1), (97, 3), (129, 2)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("split_bf16", 1e-9)])
def test_mp2_energy_of_random_integrals(n, o, precision, tol):
    """Integrals of eight decades, so that rows differ in scale.  FP64: 62 bits of every
    row's scale and exact sums, against numpy's own rounding of four sums of n terms;
    mixed: 42 bits (2.3e-13) of a row's scale through four products, with up to n terms
    of that scale in an integral: 1e-9 of the sum of magnitudes covers both."""
    rng = np.random.default_rng(100 * n + o)
    m = n * (n + 1) // 2
    k = m * (m + 1) // 2
    ints = rng.standard_normal(k) * 10.0 ** (-8.0 * rng.random(k))
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((n, n)))[0])
    lam = np.sort(np.concatenate([rng.uniform(-20.0, -0.5, o), rng.uniform(0.5, 4.0, n - o)]))
    want, scale = _energy(n, o, ints, C, lam)
    assert abs(hf.mp2_energy(ints, C, lam, o, precision=precision) - want) < tol * scale
