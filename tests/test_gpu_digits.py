"""The sliced GEMM with a chosen number of digits (hfgpu_dgemm_digits): exact sums of the
digits' products up to the longest K, and what happens when its waits run out."""
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


SCALE = {6: 42, 9: 62}  # an element is the integer sum_t d_t 128^(digits - 1 - t) times 2^-SCALE


def _elements(D, digits):
    """Doubles in (-1, 1) of digits D[..., t]; all exact."""
    Y = np.zeros(D.shape[:-1], dtype=object)
    for t in range(digits):
        Y = Y * 128 + D[..., t].astype(object)
    x = Y.astype(np.float64)
    assert np.all(x.astype(object) == Y)
    return np.ldexp(x, -SCALE[digits])


def _kept(Da, Db, digits):
    """The sum over the kept products (i + j < digits), rounded once to FP64."""
    S = np.zeros((Da.shape[0], Db.shape[1]), dtype=object)
    largest = 0
    for t in range(digits):
        g = sum(Da[:, :, i] @ Db[:, :, t - i] for i in range(t + 1))
        largest = max(largest, int(np.max(np.abs(g))))
        S = S * 128 + g.astype(object)
    assert largest < 2 ** 24
    return S.astype(np.float64) * 2.0 ** (7 * (digits - 1) - 2 * SCALE[digits]), largest


def _worst(digits, rows, K):
    """Every digit at its lowest.  With nine digits an FP64 element has no more than 53
    bits, so the last digit is 0 beside a first one; or the first is 0 beside a last one, with
    one element in K that keeps the scale."""
    if digits == 6:
        return [np.tile([-127] + [-64] * 5, (rows, K, 1))]
    top = np.tile([-63] + [-64] * 7 + [0], (rows, K, 1))
    low = np.tile([0] + [-64] * 8, (rows, K, 1))
    low[:, K // 2] = top[:, 0]
    return [top, low]


@pytest.mark.parametrize("digits,K,N,least", [(6, 512, 80, 0.99), (6, 512, 37, 0.99), (9, 455, 48, 0.77), (9, 455, 100, 0.77)])
def test_the_largest_sums_are_exact(digits, K, N, least):
    """The largest sums of digit products that FP64 operands lead to, 0.996 and 0.78 to 0.89 of
    the 2^24 below which FP32 accumulation is exact: the result is the integer sum of the
    kept products, rounded once."""
    for Da in _worst(digits, 130, K):
        for Db in _worst(digits, N, K):
            A, B = _elements(Da, digits), _elements(Db, digits).T
            want, largest = _kept(Da, Db.transpose(1, 0, 2), digits)
            rc, C = gemm(A, B, digits)
            assert rc == 0 and np.array_equal(C, want)
            assert largest > least * 2 ** 24


@pytest.mark.parametrize("digits,M,N,K", [(6, 200, 81, 512), (9, 200, 49, 455), (9, 129, 16, 31), (6, 129, 40, 33)])
def test_random_digits_are_summed_exactly(digits, M, N, K):
    """Random digits, the first element of every row at the top of its scale."""
    rng = np.random.default_rng(K + N)

    def draw(rows):
        D = rng.integers(-64, 64, (rows, K, digits))
        if digits == 9:
            D[..., 7:] = 0  # 49 bits
            D[..., 0] = rng.integers(-63, 63, (rows, K))
        D[:, 0, 0] = 126 if digits == 6 else 62
        return D

    Da, Db = draw(M), draw(N)
    want, _ = _kept(Da, Db.transpose(1, 0, 2), digits)
    rc, C = gemm(_elements(Da, digits), _elements(Db, digits).T, digits)
    assert rc == 0 and np.array_equal(C, want)
