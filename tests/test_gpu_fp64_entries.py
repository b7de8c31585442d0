"""Entries of the plain FP64 transform that digits cannot hold: what the four contractions
of transform_int2 give in FP64, entry by entry."""
import numpy as np
import pytest

import hfsolver_gb300 as hf

pytestmark = pytest.mark.gpu


def _pairs(n, int2):
    m = n * (n + 1) // 2
    M = np.zeros((m, m), dtype=int2.dtype)
    k, l = np.tril_indices(m)
    M[k, l] = int2
    M[l, k] = int2
    return M


def _transform(n, int2, C):
    """Packed MO integrals by the four contractions one after the other, plain sums in the
    operands' type."""
    i = np.arange(n)
    hi, lo = np.maximum(i[:, None], i[None, :]), np.minimum(i[:, None], i[None, :])
    pair = hi * (hi + 1) // 2 + lo
    with np.errstate(all="ignore"):
        X = _pairs(n, int2)[:, pair]  # [p][la][si]
        Y = (X[:, :, :, None] * C[None, None, :, :]).sum(2)  # [p][la][j]
        Z = (Y[:, :, :, None] * C[None, :, None, :]).sum(1)  # [p][j][b]
        W = (Z[pair][:, :, :, :, None] * C[None, :, None, None, :]).sum(1)  # [mu][j][b][i]
        T = (W[:, :, :, :, None] * C[:, None, None, None, :]).sum(0)  # [j][b][i][a]
    a, b = np.tril_indices(n)
    k, l = np.tril_indices(len(a))
    # the packed element (ij|kl), ij >= kl, is taken from T[i][j][k][l]
    return T[a[k], b[k], a[l], b[l]]


def _got(route, n, int2, C):
    """The packed MO integrals by transform_int2, or from the transform with nine digits."""
    if route == "call":
        return hf.transform_int2(int2, C)
    T = hf.half_transform(int2, C, n, 9)
    a, b = np.tril_indices(n)
    k, l = np.tril_indices(len(a))
    return T[a[k], b[k], a[l], b[l]]


@pytest.mark.parametrize("n,route", [(3, "call"), (3, "digits"), (18, "digits"), (21, "digits"), (30, "call")])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["int2", "C", "both"])
def test_nan_and_inf_go_through(n, route, bad, where):
    """An Inf or a NaN reaches the same outputs with the same values as in FP64 sums, zeros
    of C included (0 Inf is a NaN); an entry without one is left as it is."""
    rng = np.random.default_rng(n)
    m = n * (n + 1) // 2
    int2 = rng.standard_normal(m * (m + 1) // 2)
    C = np.linalg.qr(rng.standard_normal((n, n)))[0]
    C[0, n // 2] = 0.0
    if where != "C":
        int2[int2.size // 3] = bad
    if where != "int2":
        C[n - 1, n - 2] = bad
    want, got = _transform(n, int2, C), _got(route, n, int2, C)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isinf(got), np.isinf(want))
    inf = np.isinf(want)
    assert np.array_equal(got[inf], want[inf])
    ok = np.isfinite(want)
    # n 2^-52 of the largest integral times sums of n entries of C in each of four steps
    assert np.all(np.abs(got[ok] - want[ok]) <= 4 * n * 2.0 ** -52 * 8 * n * n)


def test_nan_reaches_the_fp64_energy():
    n = 37
    m = n * (n + 1) // 2
    rng = np.random.default_rng(5)
    int2 = rng.standard_normal(m * (m + 1) // 2)
    int2[100] = np.nan
    C = np.linalg.qr(rng.standard_normal((n, n)))[0]
    lam = np.sort(rng.standard_normal(n))
    assert np.isnan(hf.mp2_energy(int2, C, lam, 5))


def test_a_step_that_overflows_stays_infinite():
    """Integrals of 1e300 and C of 1e10: every sum beyond the largest double is Inf from
    the first step on, as in FP64, not turned back into numbers by the next."""
    n = 29
    m = n * (n + 1) // 2
    out = hf.transform_int2(np.full(m * (m + 1) // 2, 1e300), np.full((n, n), 1e10))
    assert np.all(np.isposinf(out))


def _fragments(rng, n):
    """Two halves 1e-7 of each other in every index and C without a block between them."""
    i, j = np.tril_indices(n)
    h = n // 2
    s = np.where(i < h, 1.0, 1e-7) * np.where(j < h, 1.0, 1e-7)
    k, l = np.tril_indices(len(i))
    C = np.zeros((n, n))
    C[:h, :h] = np.linalg.qr(rng.standard_normal((h, h)))[0]
    C[h:, h:] = np.linalg.qr(rng.standard_normal((n - h, n - h)))[0]
    return rng.uniform(0.5, 1.0, len(k)) * s[k] * s[l], C


def _graded(rng, n):
    """Integrals of sixteen decades and coefficients of twelve, without an order."""
    m = n * (n + 1) // 2
    k = m * (m + 1) // 2
    return rng.standard_normal(k) * 10.0 ** (-16.0 * rng.random(k)), rng.standard_normal((n, n)) * 10.0 ** (-12.0 * rng.random((n, n)))


def _scaled(a, c):
    def make(rng, n):
        m = n * (n + 1) // 2
        return a * rng.standard_normal(m * (m + 1) // 2), c * rng.standard_normal((n, n))
    return make


@pytest.mark.parametrize("make", [_fragments, _graded, _scaled(1e-290, 1.0), _scaled(1e-150, 1e-35), _scaled(3e-320, 1e5),
                                  _scaled(1e280, 1e2), _scaled(1.0, 1.0)],
                         ids=["fragments", "graded", "tiny", "small", "subnormal", "huge", "plain"])
@pytest.mark.parametrize("n,route", [(6, "call"), (6, "digits"), (18, "digits"), (25, "digits"), (29, "call")])
def test_every_entry_is_as_good_as_an_fp64_sum(n, route, make):
    """Against extended precision, entry by entry: four sums of n terms, each within n 2^-53
    of the sum of the terms' magnitudes (twice that covers products of the four factors),
    and half the smallest subnormal for each product that underflows, through the steps
    that follow it."""
    int2, C = make(np.random.default_rng(n), n)
    got = _got(route, n, int2, C).astype(np.longdouble)
    X, D = int2.astype(np.longdouble), C.astype(np.longdouble)
    want, scale = _transform(n, X, D), _transform(n, np.abs(X), np.abs(D))
    q = n * np.longdouble(np.max(np.abs(C)))
    under = n * np.longdouble(2.0 ** -1074) * (1 + q + q * q + q * q * q)
    assert np.all(np.abs(got - want) <= 8 * n * np.longdouble(2.0 ** -53) * scale + under)


@pytest.mark.parametrize("n", [4, 15, 24])
def test_small_transforms_launch_no_cutting_kernels(n):
    """A small basis takes the kernels of the FP64 GEMM transform alone."""
    from hfsolver_gb300 import _lib

    L = _lib.lib()
    m = n * (n + 1) // 2
    int2, C = np.ones(m * (m + 1) // 2), np.eye(n)
    k = [L.hfgpu_kernel_launches()]
    hf.half_transform(int2, C, n, 0)
    k.append(L.hfgpu_kernel_launches())
    hf.transform_int2(int2, C)
    k.append(L.hfgpu_kernel_launches())
    assert k[2] - k[1] == k[1] - k[0] + 1  # and the packing


@pytest.mark.parametrize("n,o", [(25, 5), (30, 6), (35, 17)])
def test_small_half_transforms_launch_no_cutting_kernels(n, o):
    from hfsolver_gb300 import _lib

    L = _lib.lib()
    m = n * (n + 1) // 2
    int2, C = np.ones(m * (m + 1) // 2), np.eye(n)
    k = [L.hfgpu_kernel_launches()]
    hf.half_transform(int2, C, o, 0)
    k.append(L.hfgpu_kernel_launches())
    hf.mp2_energy(int2, C, np.arange(n) - o + 0.5, o)
    k.append(L.hfgpu_kernel_launches())
    assert k[2] - k[1] == k[1] - k[0] + 1  # and the energy
