"""Integrals whose primitive pairs are shared by more or fewer lanes with the size of
the molecule: few shell pairs or quartets, and enough of them to fill the GPU."""
import numpy as np
import pytest

import hfsolver_gb300 as hf
from tests.gpu_common import assert_close, basis_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [1, 3, 10])
def test_integrals_small_and_large(oracle, nw):
    """S, T, V against the oracle, and the first water's electron repulsion integrals
    against the ones computed for it alone.  The tolerances are those of the other
    comparisons with the oracle: sums of at most 36^2 primitive terms, each good to a
    few units of roundoff of its size, and V over 30 nuclei of charge up to 8."""
    from hfsolver_gb300.clusters import water_cluster

    atno, xyz = water_cluster(nw, seed=31, jitter=0.02)
    b = oracle.Basis(atno, xyz)
    args = basis_args(b)
    assert_close(hf.getS(*args), oracle.one_electron(b, "S"), 1e-12, 1e-12, "S")
    assert_close(hf.getT(*args), oracle.one_electron(b, "T"), 1e-12, 1e-12, "T")
    V = hf.getV(*args, b.atno, b.xyz[:, 0], b.xyz[:, 1], b.xyz[:, 2])
    assert_close(V, oracle.one_electron(b, "V"), 1e-11, 1e-12, "V")
    b1 = oracle.Basis(atno[:3], xyz[:3])
    alone = hf.getInts(*basis_args(b1))  # packed: the first functions' integrals lead the array
    assert_close(hf.getInts(*args)[:alone.size], alone, 1e-12, 1e-12, "ERI")
