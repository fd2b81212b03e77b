"""The warp that finds nodes and weights, with its lanes run in different
orders between the warp's primitives: no lane may read an entry that another
one writes meanwhile, so every order gives the same bits, and the bits are the
eigenvalues.

Tolerance: implicit QL is backward stable, eigenvalues of a k x k matrix are
within about k * eps * |T| (k <= 100: 3e-14); 1e-12 is used, as for the
kernel."""

import ctypes

import numpy as np
import pytest
from scipy.linalg import eigh_tridiagonal

import native


@pytest.fixture(scope="module")
def ql(tmp_path_factory):
    return native.load("ql_warp", tmp_path_factory.mktemp("ql")).ql_warp


def _solve(ql, alpha, beta, order):
    d, e = alpha.copy(), np.append(beta, 0.0)
    z = np.zeros(alpha.size)
    z[0] = 1.0
    dp = ctypes.POINTER(ctypes.c_double)
    o = (ctypes.c_int * 32)(*order)
    races = ctypes.c_long(-1)
    st = ql(*[v.ctypes.data_as(dp) for v in (d, e, z)], alpha.size, o,
            ctypes.byref(races))
    assert races.value == 0
    return st, d, e, z


@pytest.mark.parametrize("k", [2, 3, 20, 33, 100])
@pytest.mark.parametrize("split", [False, True])
def test_every_order_of_the_lanes_gives_the_same_nodes(ql, k, split):
    g = np.random.default_rng(k)
    alpha = 1.5 + 2.0 * g.random(k)
    beta = 0.5 * g.random(k - 1)
    if split:
        beta[(k - 1) // 2] = 0.0
    orders = [list(range(32)), list(range(31, -1, -1)),
              list(g.permutation(32))]
    runs = [_solve(ql, alpha, beta, o) for o in orders]
    for st, d, e, z in runs:
        assert st == 0
        for got, want in zip((d, e, z), runs[0][1:]):
            assert np.array_equal(got, want)
    want = eigh_tridiagonal(alpha, beta, eigvals_only=True)
    assert np.max(np.abs(np.sort(runs[0][1]) - want)) < 1e-12 * want[-1]
    assert abs(np.sum(runs[0][3]**2) - 1.0) < 1e-12
