"""The Fock digest against J and K of the same integrals in plain numpy, at sizes where
its classes leave ragged warps and its row splits change, full and screened."""
import numpy as np
import pytest

import hfsolver_gb300 as hf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,incremental,autotune", [(1, False, False), (1, True, False), (2, False, False),
                                                     (3, True, False), (3, False, True), (5, True, False)])
def test_scf_energy_from_the_digest(nw, incremental, autotune):
    """E0 = tr P (H + F) / 2 of the converged density, with F from formG over unscreened
    packed integrals: the digest only enters through the SCF that found the density.
    Tolerance: the SCF stops at dP < 1e-10, the energy's error is of second order, and
    |E0| < 600 with sums of ~1e5 terms of unit roundoff 1.1e-16: 1e-10 covers both."""
    from hfsolver_gb300.clusters import water_cluster
    from oracle import oracle as O
    from tests.gpu_common import basis_args

    atno, xyz = water_cluster(nw, seed=21 + nw, jitter=0.02)
    b = O.Basis(atno, xyz)
    r = hf.rhf(atno, xyz, hf.RHFOptions(nscf=100, diis=True, schwarz=1e-13, tolP=1e-10, tolE=1e-12, mp2="none",
                                        incremental=incremental, autotune=autotune, guess="sad"), want_orbitals=True)
    Co = r["C"][:, :r["nocc"]]
    P = 2.0 * Co @ Co.T
    T = hf.getT(*basis_args(b))
    V = hf.getV(*basis_args(b), b.atno, *np.ascontiguousarray(b.xyz.T))
    G = hf.formG(P, hf.getInts(*basis_args(b)))
    E0 = float(np.sum(P * (T + V)) + 0.5 * np.sum(P * G))
    assert abs(E0 - r["E0"]) < 1e-10
