"""Nodes and weights (one warp per probe) and the quadrature (one warp per
probe and inquiry) at the sizes where their loops change shape: one to three
passes of 32 lanes over the nodes, the smallest and largest degrees, probes
that stopped early, entries whose squares leave the range of a double, and
several inquiries.

Tolerance: implicit QL is backward stable, so eigenvalues of a k x k matrix
are within about k * eps * |T| (k <= 256: 6e-14) and the quadrature of
1/x over a spectrum in [0.5, 4.5] within ten times that: 1e-12 is used for
both."""

import ctypes

import numpy as np
import pytest
from scipy.linalg import eigh_tridiagonal

import imate_b200 as ib
from imate_b200 import _lib

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _solve(cuda, alpha, beta, sizes, gram=0):
    import torch
    m, b = alpha.shape
    a, bt = torch.from_numpy(alpha).cuda(), torch.from_numpy(beta).cuda()
    sz = torch.from_numpy(sizes.astype(np.int32)).cuda()
    th = torch.zeros((m, b), dtype=torch.float64, device="cuda")
    ta = torch.zeros_like(th)
    st = torch.full((b,), -1, dtype=torch.int32, device="cuda")
    _lib.check(cuda.slq_nodes_weights(
        a.data_ptr(), bt.data_ptr(), sz.data_ptr(), b, m, gram, th.data_ptr(),
        ta.data_ptr(), st.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return th.cpu().numpy(), ta.cpu().numpy(), st.cpu().numpy()


@pytest.mark.parametrize("scale", [1.0, 1e-200, 1e200])
@pytest.mark.parametrize("m", [1, 2, 3, 31, 32, 33, 64, 65, 255, 256])
def test_nodes_and_weights_at_every_loop_edge(cuda, m, scale):
    g = np.random.default_rng(m)
    b = 5
    alpha = (1.5 + 2.0 * g.random((m, b))) * scale
    beta = 0.5 * g.random((m, b)) * scale
    sizes = np.array([m, max(1, m - 1), max(1, m // 2), 1, m])
    th, ta, st = _solve(cuda, alpha, beta, sizes)
    assert np.all(st == 0)
    for p in range(b):
        k = sizes[p]
        # the reference works on the matrix scaled back to 1
        want, Q = eigh_tridiagonal(alpha[:k, p] / scale,
                                   beta[:k - 1, p] / scale)
        at = np.argsort(th[:k, p])
        got = th[at, p] / scale
        assert np.max(np.abs(got - want)) < TOL * np.max(np.abs(want))
        assert abs(np.sum(ta[:k, p]**2) - 1.0) < TOL
        quad = np.sum(ta[at, p]**2 / got)
        ref = np.sum(Q[0]**2 / want)
        assert abs(quad - ref) < TOL * abs(ref)


def test_zero_and_nonfinite_matrices_are_reported(cuda):
    alpha = np.zeros((40, 4))
    beta = np.zeros((40, 4))
    alpha[:, 1] = 2.0
    alpha[7, 2] = np.nan
    alpha[:, 3] = 1.0
    beta[3, 3] = np.inf
    th, ta, st = _solve(cuda, alpha, beta, np.full(4, 40))
    assert list(st[:2]) == [0, 0]
    assert np.all(th[:, 0] == 0.0) and np.all(th[:, 1] == 2.0)
    assert st[2] & 1 and st[3] & 1


@pytest.mark.parametrize("degree,q", [(1, 1), (31, 3), (33, 40), (70, 9)])
def test_every_inquiry_equals_its_own_run(cuda, degree, q):
    """Inquiry j of a sweep is the run with t_0's Krylov coefficients shifted
    to t_j: within rounding of a call with t_j alone (full
    reorthogonalisation, float64)."""
    A = ib.correlation_matrix(700, scale=0.05, shift=0.3, seed=degree)
    t = np.linspace(0.0, 3.0, q)
    kw = dict(method="slq", gpu=True, return_info=True, min_num_samples=5,
              max_num_samples=5, error_rtol=0.0, lanczos_degree=degree,
              orthogonalize=-1, seed=4)
    Aop = ib.AffineMatrixFunction(A)
    _, info = ib.logdet(Aop, parameters=t, **kw)
    got = np.asarray(info["convergence"]["samples"]).reshape(5, q)
    for j in (0, q // 2, q - 1):
        _, one = ib.logdet(Aop, parameters=float(t[j]), **kw)
        want = np.asarray(one["convergence"]["samples"])
        assert np.max(np.abs(got[:, j] - want) / np.abs(want)) < 1e-10
