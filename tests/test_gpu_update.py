"""The update passes (three-term update without a basis, and the one that takes
the basis out) where their 16-byte pieces end: one and two probes, rows around
a piece and around a whole wave of CTAs, blocks wider than 256 probes, and
every remainder of the basis vectors loaded at once.  Float64 samples within
1e-10 of the oracle (the parity bar), float32 within 1e-6 n / |sample| of it
(the mixed-precision bar, relative to the terms of the sum)."""

import numpy as np
import pytest

import imate_b200 as ib
from oracle import oracle

pytestmark = pytest.mark.gpu


# rows of a piece: 1024 (float64) or 2048 (float32) values over the probes
@pytest.mark.parametrize("block,n", [(1, 1023), (1, 1025), (1, 3), (2, 1),
                                     (2, 1023), (2, 2049), (4, 513),
                                     (64, 15), (64, 33), (64, 4800),
                                     (256, 5), (512, 9), (512, 1201)])
@pytest.mark.parametrize("orth", [0, -1])
def test_pieces(cuda, block, n, orth):
    if n > 3:
        A = ib.correlation_matrix(n, scale=min(0.5, 0.6 / np.sqrt(n)),
                                  shift=0.3, seed=n)
    else:
        import scipy.sparse as sp
        A = sp.csr_matrix(2.0 * np.eye(n) + 0.1)
    count = min(block, 3)
    for degree in {min(n, d) for d in (2, 5, 8, 11)}:
        kw = dict(error_rtol=0.0, lanczos_degree=degree, orthogonalize=orth,
                  seed=5)
        ref = oracle.trace_estimator(A, "log", gram=False,
                                     min_num_samples=count,
                                     max_num_samples=count,
                                     **kw)["samples"][:count, 0]
        for dtype, bar in ((np.float64, 1e-10), (np.float32, 1e-6)):
            _, info = ib.logdet(
                ib.Matrix(A.astype(dtype), reorder=False, group_rows=0),
                method="slq", gpu=True, return_info=True, block_size=block,
                min_num_samples=block, max_num_samples=block, **kw)
            got = np.asarray(info["convergence"]["samples"], float)[:count]
            tol = bar * (np.abs(ref) if dtype == np.float64 else
                         np.maximum(np.abs(ref), n))
            assert np.all(np.abs(got - ref) <= tol)
