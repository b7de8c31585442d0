"""The gather-fed sliced GEMM at the edges of its tiles: one and two accumulator sets, the
40-column tile whose products are padded, K below one 16-step and with a ragged end,
rows past a tile, several column tiles, zero and subnormal rows, odd strides."""
import numpy as np
import pytest

from tests.test_gpu_tcgemm import sliced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (129, 5, 15), (127, 16, 17), (128, 33, 25), (700, 40, 200), (257, 41, 33),
                                   (300, 80, 511), (40000, 48, 64), (513, 81, 47), (260, 163, 129)])
def test_sliced_gemm_tile_edges(M, N, K):
    """Tolerance: 2^-40 K of the row's and column's largest entries, from entries kept to
    2^-42 of a power of two that is at most twice the largest."""
    rng = np.random.default_rng(1000 * N + K)
    A = rng.standard_normal((M, K)) * 10.0 ** rng.uniform(-6, 6, size=(M, 1))
    B = rng.standard_normal((K, N)) * 10.0 ** rng.uniform(-3, 3, size=(1, N))
    if M > 100:
        A[3] = 0.0
        A[5] = 1e-310
        A[7, 1:] *= 1e-30
    if N > 4:
        B[:, 2] = 0.0
    C = sliced(A, B)
    bound = 2.0 ** -40 * K * np.max(np.abs(A), axis=1)[:, None] * np.max(np.abs(B), axis=0)[None, :] + 1e-300
    assert np.all(np.abs(C - A @ B) <= bound)


def test_sliced_gemm_exact_where_digits_agree():
    """Equal digits of one sign everywhere are the largest sums the FP32 accumulators
    meet; 512 products of (1 - 2^-42)^2 are kept exactly by six digits per factor down to
    the last group, so the result is within 512 2^-42 of it relative to 512."""
    x = 1.0 - 2.0 ** -42
    C = sliced(np.full((130, 512), x), np.full((512, 80), -x))
    assert np.all(np.abs(C + 512.0 * x * x) <= 512.0 * 2.0 ** -41)


@pytest.mark.parametrize("n,seed", [(3, 0), (17, 1), (26, 2)])
def test_fp64_transform_against_extended_precision(n, seed):
    """transform_int2 with nine digits per factor against the same contraction in extended
    precision.  Each of the four steps keeps its sums to 2^-62 n of the factors' scales and
    rounds once to FP64 (2^-53), with intermediate values at most n times the largest
    integral (orthogonal C): 4 n 2^-52 of the largest result and integral bounds it."""
    import hfsolver_gb300 as hf

    rng = np.random.default_rng(seed)
    m = n * (n + 1) // 2
    B = rng.standard_normal((m, n)) * 10.0 ** rng.uniform(-4, 0, size=(m, 1))
    M = B @ B.T
    k, l = np.tril_indices(m)
    int2 = np.ascontiguousarray(M[k, l])
    C = np.linalg.qr(rng.standard_normal((n, n)))[0]
    out = hf.transform_int2(int2, C)
    M = np.zeros((m, m))
    M[k, l] = int2
    M[l, k] = int2
    i, j = np.tril_indices(n)
    X, Cl = M.astype(np.longdouble), C.astype(np.longdouble)
    for _ in range(2):
        Q = np.zeros((m, n, n), dtype=np.longdouble)
        Q[:, i, j] = X
        Q[:, j, i] = X
        X = np.ascontiguousarray(np.stack([Cl.T @ (q @ Cl) for q in Q])[:, i, j].T)
    err = np.max(np.abs((out - X[k, l]).astype(np.float64)))
    assert err <= 4 * n * 2.0 ** -52 * max(np.max(np.abs(int2)), float(np.max(np.abs(X))))
