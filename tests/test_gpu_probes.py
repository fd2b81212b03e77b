"""Parity probes at the edges of their generator: one chunk and many, chunk
and jump-table boundaries (16 words a chunk, 16 chunks a table step), widths
that fill no quad or no 64-probe tile, one-element rows, and blocks whose
start states are jumped to on the device.  Bit for bit against the oracle's
stream."""

import ctypes

import numpy as np
import pytest

import imate_b200 as ib
from imate_b200 import _lib
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,count", [(1, 1), (3, 2), (4, 4), (50, 49),
                                         (64, 64), (100, 97), (130, 130)])
@pytest.mark.parametrize("n", [1, 63, 64, 4095, 4096, 4097, 5119, 16383,
                               16384, 17000])
def test_probes_bit_exact_at_chunk_edges(cuda, n, width, count):
    import torch
    want = oracle.random_probes(9, n, count + 2)[2:]
    nb = ctypes.c_size_t(0)
    _lib.check(cuda.slq_generate_probes_workspace_bytes(n, width,
                                                        ctypes.byref(nb)))
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    for code, dt in ((_lib.SLQ_F32, torch.float32),
                     (_lib.SLQ_F64, torch.float64)):
        out = torch.full((n, width), 7.0, dtype=dt, device="cuda")
        _lib.check(cuda.slq_generate_probes(
            9, 0, n, 2, count, width, code, out.data_ptr(), ws.data_ptr(),
            ws.numel(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert np.array_equal(got[:, :count].T, want)
        assert np.all(got[:, count:] == 0.0)


@pytest.mark.parametrize("block", [1, 16, 32, 64])
def test_blocks_continue_the_stream(cuda, block):
    """Every block of a run starts where the last one ended: trace(A) of a
    dense-ish float64 matrix by one-step quadrature is z^T A z of each probe,
    whatever the block width."""
    n = 300
    A = ib.correlation_matrix(n, scale=0.1, shift=0.3, seed=1)
    _, info = ib.trace(A, method="slq", gpu=True, return_info=True,
                       min_num_samples=70, max_num_samples=70,
                       error_rtol=0.0, lanczos_degree=2, orthogonalize=0,
                       seed=9, block_size=block)
    Z = oracle.random_probes(9, n, 70)
    want = np.einsum("pi,pi->p", Z, (A @ Z.T).T)
    got = np.asarray(info["convergence"]["samples"])
    assert np.max(np.abs(got - want) / np.abs(want)) < 1e-12
