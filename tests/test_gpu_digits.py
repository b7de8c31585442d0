"""The sliced GEMM with a chosen number of digits (hfgpu_dgemm_digits): what happens when
its waits run out."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gemm(A, B, digits, spins=-1):
    """(status, A B)"""
    from hfsolver_gb300 import _lib

    A, Bt = np.ascontiguousarray(A), np.ascontiguousarray(B.T)
    (M, K), N = A.shape, B.shape[1]
    C = np.zeros((M, N))
    dp = ctypes.POINTER(ctypes.c_double)
    rc = _lib.lib().hfgpu_dgemm_digits(M, N, K, A.ctypes.data_as(dp), Bt.ctypes.data_as(dp), C.ctypes.data_as(dp), digits,
                                       spins)
    return rc, C


# one and two sets of accumulators; less than a pipeline of steps, several tiles per CTA
@pytest.mark.parametrize("M,N,K", [(100, 16, 20), (128, 40, 400), (30000, 48, 100), (30000, 16, 70)])
@pytest.mark.parametrize("digits", [6, 9])
def test_a_wait_that_runs_out_is_reported(M, N, K, digits):
    """Every block leaves after its first wait, and the next product is right: integers
    that both kinds of digits hold."""
    from hfsolver_gb300 import _lib

    rng = np.random.default_rng(M + N)
    A, B = rng.integers(-50, 50, (M, K)).astype(float), rng.integers(-50, 50, (K, N)).astype(float)
    rc, _ = gemm(A, B, digits, 0)
    assert rc == _lib.ERR_CUDA and b"timed out" in _lib.lib().hfgpu_last_error()
    rc, C = gemm(A, B, digits)
    assert rc == _lib.OK and np.array_equal(C, A @ B)
