"""The dense product's BF16 parts and K chunks at the edges of its tiles, on
data that spans FP32's range, and with non-finite entries.

The bound on |Y - A X| is per element, in units of S = |A| |X|: the products
left out are below 2^-22 S; a 64-value chunk takes 24 MMAs, each adding 16
products to the accumulator with an error of at most 2^-22 of its magnitude,
24 * 2^-22 < 2^-17 S; the chunks' sums and the result round to nearest, K / 64
+ 1 times 2^-24 S.  2^-16 + K / 64 * 2^-24 covers them.
"""

import numpy as np
import pytest

import imate_b200 as ib

pytestmark = pytest.mark.gpu


def _product(A, X, transpose=False):
    import torch
    op = ib.Matrix(A).get_device_operator(need_transpose=True)
    assert getattr(op, "dense", False)
    Y = op.dot(torch.from_numpy(X).cuda(), transpose=transpose)
    return Y.cpu().numpy().astype(np.float64)


def _assert_close(Y, A, X):
    A, X = A.astype(np.float64), X.astype(np.float64)
    bound = (2.0 ** -16 + A.shape[1] / 64 * 2.0 ** -24) * (np.abs(A) @ np.abs(X))
    assert np.all(np.abs(Y - A @ X) <= bound)


@pytest.mark.parametrize("rows,cols,width", [
    (1, 1, 1), (127, 31, 15), (128, 32, 16), (129, 33, 17), (128, 64, 32),
    (257, 65, 255), (200, 2049, 256), (77, 129, 257), (9601, 130, 48)])
def test_tile_edges(cuda, rows, cols, width):
    rng = np.random.default_rng(rows + 3 * cols + width)
    A = rng.standard_normal((rows, cols)).astype(np.float32)
    X = rng.standard_normal((cols, width)).astype(np.float32)
    _assert_close(_product(A, X), A, X)
    X = rng.standard_normal((rows, width)).astype(np.float32)
    _assert_close(_product(A, X, transpose=True), A.T, X)


@pytest.mark.parametrize("n", [200, 2000])
def test_wide_range(cuda, n):
    """Entries that differ by 10^24 in A, in X, and the other way round in
    both (so that the products are of one size)."""
    rng = np.random.default_rng(n)
    d = 10.0 ** rng.uniform(-12, 12, n)
    A = rng.standard_normal((n, n))
    X = rng.standard_normal((n, 40))
    for a, x in ((A * d, X), (A, X * d[:, None]), (A * d, X / d[:, None]),
                 (A * d * d[:, None], X)):
        a, x = a.astype(np.float32), x.astype(np.float32)
        _assert_close(_product(a, x), a, x)


def test_largest_values(cuda):
    """FP32's largest value is above BF16's; it stays finite."""
    rng = np.random.default_rng(0)
    A = np.full((130, 70), np.finfo(np.float32).max, dtype=np.float32)
    A[:, ::2] *= -1
    X = (1e-6 * rng.standard_normal((70, 20))).astype(np.float32)
    _assert_close(_product(A, X), A, X)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite_rows(cuda, value):
    """A non-finite entry spoils its row (or, in X, its probe) and no other."""
    rng = np.random.default_rng(1)
    A = rng.standard_normal((300, 200)).astype(np.float32)
    X = rng.standard_normal((200, 24)).astype(np.float32)
    A[131, 64] = value
    X[199, 7] = value
    Y = _product(A, X)
    assert not np.isfinite(Y[131]).any() and not np.isfinite(Y[:, 7]).any()
    rows = np.arange(300) != 131
    probes = np.arange(24) != 7
    _assert_close(Y[rows][:, probes], A[rows], X[:, probes])
