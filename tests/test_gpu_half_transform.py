"""The three transforms to (ia|jb), FP64 GEMMs and sliced GEMMs with nine and six digits,
each against plain sums and against each other, at sizes where one molecule would take
only one of them."""
import numpy as np
import pytest

import hfsolver_gb300 as hf

pytestmark = pytest.mark.gpu


def _input(n, seed):
    rng = np.random.default_rng(seed)
    m = n * (n + 1) // 2
    int2 = rng.standard_normal(m * (m + 1) // 2)
    return int2, np.asfortranarray(np.linalg.qr(rng.standard_normal((n, n)))[0])


def _sums(n, int2, C, o):
    """T[j][b][i][a] by the four contractions in numpy, in the operands' type."""
    i = np.arange(n)
    hi, lo = np.maximum(i[:, None], i[None, :]), np.minimum(i[:, None], i[None, :])
    pair = hi * (hi + 1) // 2 + lo
    m = n * (n + 1) // 2
    M = np.zeros((m, m), dtype=int2.dtype)
    k, l = np.tril_indices(m)
    M[k, l] = int2
    M[l, k] = int2
    C1, C2 = C[:, :o], C[:, o:] if o < n else C
    Z = np.einsum("plj,lb->pjb", np.einsum("pls,sj->plj", M[:, pair], C1), C2)
    return np.einsum("mjbi,ma->jbia", np.einsum("mnjb,ni->mjbi", Z[pair], C1), C2)


# one function; below, at and past the 8 pairs and 16 indices of a row block, the 128 rows of
# a tile and the 16 and 32 k of a step; all columns on both sides
@pytest.mark.parametrize("n,o", [(1, 1), (2, 1), (7, 3), (8, 8), (15, 14), (17, 1), (33, 16), (34, 5)])
@pytest.mark.parametrize("path", [0, 9])
def test_against_extended_precision(n, o, path):
    """Four sums of n terms, each within n 2^-53 of the sum of the terms' magnitudes: twice
    4 n 2^-53 of that through all four (the other half for the products of the factors)."""
    int2, C = _input(n, 10 * n + o)
    X, D = int2.astype(np.longdouble), C.astype(np.longdouble)
    got = hf.half_transform(int2, C, o, path)
    assert np.all(np.abs(got - _sums(n, X, D, o)) <= 8 * n * np.longdouble(2.0 ** -53) * _sums(n, np.abs(X), np.abs(D), o))


# several blocks of pairs and of (j, b), an odd size; rows of more than 256 elements
@pytest.mark.parametrize("n,o", [(181, 90), (260, 3)])
def test_digits_against_fp64_gemms(n, o):
    """Nine digits: entry by entry, both within 8 n 2^-53 of the terms' magnitudes.  Six: a
    step keeps 2^-40 n of the largest factors (see the GEMM's own tests), and each later one
    grows it by n of C's largest entry."""
    int2, C = _input(n, n)
    ref = hf.half_transform(int2, C, o, 0)
    scale = hf.half_transform(np.abs(int2), np.abs(C), o, 0)
    assert np.all(np.abs(hf.half_transform(int2, C, o, 9) - ref) <= 16 * n * 2.0 ** -53 * scale)
    bound = 4 * 2.0 ** -40 * np.max(np.abs(int2)) * (n * np.max(np.abs(C))) ** 4
    assert np.max(np.abs(hf.half_transform(int2, C, o, 6) - ref)) <= bound
