"""Nuclear attraction of very many centres on a small basis, as an embedding in point charges
asks for: more of them than a launch has block rows."""
import numpy as np
import pytest

import hfsolver_gb300 as hf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nat", [65534, 65535, 70001, 262140])
def test_v_of_many_centres(nat):
    """V is a sum over the centres: that of all of them against that of their parts, to the
    roundoff of sums of nat terms of one sign."""
    rng = np.random.default_rng(nat)
    args = ([1, 1], [0, 1], [0.0, 0.0], [0.0, 0.3], [0.0, -0.2], [0, 1], [0, 0], [0, 0], [0.7, 0.5], [1.1, 0.6])
    z = rng.integers(1, 9, nat).astype(np.int32)
    x = rng.uniform(-40.0, 40.0, (3, nat))
    whole = hf.getV(*args, z, *x)
    parts = sum(hf.getV(*args, z[k:k + 10000], *x[:, k:k + 10000]) for k in range(0, nat, 10000))
    assert np.all(np.abs(whole - parts) <= nat * 2.0 ** -52 * np.max(np.abs(np.diag(whole))))
    assert whole[0, 0] < -1000.0
