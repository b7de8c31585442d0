"""Results that do not change from call to call."""
import numpy as np
import pytest

import hfsolver_gb300 as hf
from tests.gpu_common import basis_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [1, 2, 4])
def test_nuclear_attraction_to_the_bit(oracle, nw):
    """The nuclei's parts of V are formed side by side and summed in a fixed order."""
    from hfsolver_gb300.clusters import water_cluster

    b = oracle.Basis(*water_cluster(nw, seed=8, jitter=0.02))
    args = basis_args(b) + (b.atno, b.xyz[:, 0], b.xyz[:, 1], b.xyz[:, 2])
    first = hf.getV(*args)
    assert all(np.array_equal(hf.getV(*args), first) for _ in range(60))
