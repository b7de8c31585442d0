"""A call that fails half-way leaves nothing behind for the next."""
import numpy as np
import pytest

import hfsolver_gb300 as hf
from hfsolver_gb300 import _lib
from hfsolver_gb300.clusters import water_cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "split_bf16"])
def test_gemm_counters_after_a_failed_transform(precision):
    """Each device allocation of an MBPT2 energy fails in turn, some of them between two sliced
    GEMMs: the next call counts its own GEMMs only."""
    n, o = 40, 6
    m = n * (n + 1) // 2
    rng = np.random.default_rng(2)
    int2 = rng.standard_normal(m * (m + 1) // 2)
    C = np.linalg.qr(rng.standard_normal((n, n)))[0]
    lam = np.concatenate([np.linspace(-9.0, -1.0, o), np.linspace(1.0, 3.0, n - o)])
    atno, xyz = water_cluster(1, seed=1)
    opt = hf.RHFOptions(mp2="split_bf16")
    want = hf.mp2_energy(int2, C, lam, o, precision)
    ref = hf.rhf(atno, xyz, opt)
    L = _lib.lib()
    failed = 0
    for k in range(1, 100):
        L.hfgpu_fail_allocation(k)
        try:
            got = hf.mp2_energy(int2, C, lam, o, precision)
        except hf.HFGPUError as e:
            assert e.code == _lib.ERR_NOMEM
            failed += 1
        else:
            break
        finally:
            L.hfgpu_fail_allocation(0)
        r = hf.rhf(atno, xyz, opt)
        assert r["n_tc_step1"] == ref["n_tc_step1"] and r["tc_flops"] == ref["tc_flops"]
    assert failed > 8 and got == want


@pytest.mark.parametrize("options", [dict(diis=True, mp2="fp64"), dict(diis=True, purify=True, incremental=True, guess="sad",
                                                                      schwarz=1e-12, mp2="split_bf16")])
def test_a_molecule_after_a_failed_one(options):
    """Each device allocation of a molecule's pipeline fails in turn, with integrals still
    running on the side streams for some: they are waited for, and the next molecule gets
    the energies it had before.  (They are sums of atomics: 1e-10.)"""
    big, small = water_cluster(4, seed=2), water_cluster(2, seed=3)
    opt = hf.RHFOptions(nscf=60, **options)
    ref = [hf.rhf(*m, opt) for m in (big, small)]
    L = _lib.lib()
    failed = 0
    for k in range(1, 2000):
        L.hfgpu_fail_allocation(k)
        try:
            r = hf.rhf(*big, opt)
        except hf.HFGPUError as e:
            assert e.code == _lib.ERR_NOMEM
            failed += 1
        else:
            break
        finally:
            L.hfgpu_fail_allocation(0)
        s = hf.rhf(*small, opt)
        assert abs(s["Etot"] - ref[1]["Etot"]) < 1e-10 and abs(s["E2"] - ref[1]["E2"]) < 1e-8
    assert failed > 40 and abs(r["Etot"] - ref[0]["Etot"]) < 1e-10
