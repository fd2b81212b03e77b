"""The streaming passes at row counts around their tiles: the rows past the
last whole tile are dealt over the CTAs, basis tiles are taken in pairs with a
single one left over, and the plain three-term update (no basis) is a kernel
of its own.  Float64 samples within 1e-10 of the oracle (the parity bar), for
full, windowed and no reorthogonalisation; float32 within 1e-6 of float64 on
the same probes (the mixed-precision bar)."""

import numpy as np
import pytest

import imate_b200 as ib
from oracle import oracle

pytestmark = pytest.mark.gpu


def _run(A, **kw):
    _, info = ib.logdet(A, method="slq", gpu=True, return_info=True, **kw)
    return np.asarray(info["convergence"]["samples"], float)


# float64 tiles hold 8 x 256 values: 8 rows at 256 probes, 128 at 16, 2048 at 1
@pytest.mark.parametrize("block,n", [(1, 2047), (1, 2049), (1, 6200),
                                     (16, 127), (16, 128), (16, 1407),
                                     (256, 7), (256, 9), (256, 1191)])
@pytest.mark.parametrize("orth", [0, 3, -1])
def test_rows_past_the_last_tile(cuda, block, n, orth):
    A = ib.correlation_matrix(n, scale=min(0.5, 0.6 / np.sqrt(n)), shift=0.3,
                              seed=n)
    count = 2 if block == 1 else 3
    degree = min(9, n)
    kw = dict(error_rtol=0.0, lanczos_degree=degree, orthogonalize=orth,
              seed=3)
    want = oracle.trace_estimator(A, "log", gram=False,
                                  min_num_samples=count,
                                  max_num_samples=count, **kw)
    # a block wider than the samples asked for: fill it with more samples
    got = _run(ib.Matrix(A, reorder=False, group_rows=0), block_size=block,
               min_num_samples=max(count, block),
               max_num_samples=max(count, block), **kw)[:count]
    ref = want["samples"][:count, 0]
    assert np.max(np.abs(got - ref) / np.abs(ref)) < 1e-10
    if orth == -1:
        got32 = _run(ib.Matrix(A.astype(np.float32), reorder=False,
                               group_rows=0), block_size=block,
                     min_num_samples=max(count, block),
                     max_num_samples=max(count, block), **kw)[:count]
        assert np.max(np.abs(got32 - ref) / np.abs(ref)) < 1e-6 * \
            max(1.0, n / np.min(np.abs(ref)))


def test_more_vectors_than_the_sums_of_one_pass(cuda):
    """Float64 products with more basis vectors than fit the plain-load pass
    (48), and with more than one launch takes (64)."""
    A = ib.correlation_matrix(211, scale=0.05, shift=0.3, seed=2)
    kw = dict(min_num_samples=3, max_num_samples=3, error_rtol=0.0,
              lanczos_degree=70, orthogonalize=-1, seed=3)
    want = oracle.trace_estimator(A, "log", gram=False, **kw)
    got = _run(ib.Matrix(A, reorder=False, group_rows=0), **kw)
    ref = want["samples"][:3, 0]
    assert np.max(np.abs(got - ref) / np.abs(ref)) < 1e-10
