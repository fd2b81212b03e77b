"""The CSR product of blocks of 32 probes and more (k_spmm_rows) against
float64 numpy at the sizes where its loops change shape: every block width
(rows that share a warp, one piece per lane, several), row lengths around the
number of entries gathered at once and zero, row counts below, at and above
what the warps of a block take, with and without the shift of A + t I, and
buffers that are not 16-byte aligned.

Tolerance: a row of k entries is k fused multiply-adds and at most three
more roundings, so |error| <= (k + 3) eps sum |a_i x_i| (eps of the stored
type), plus the shift's term."""

import numpy as np
import pytest
import scipy.sparse as sp

import imate_b200 as ib
from imate_b200 import _lib
from imate_b200.linear_operator import _DeviceOperator

pytestmark = pytest.mark.gpu


def _matrix(n, dtype, seed):
    """Rows of 0, 1, ... 37 entries (and one long row), columns spread."""
    g = np.random.default_rng(seed)
    lens = np.minimum(g.permutation(np.arange(n) % 38), n)
    lens[n // 2] = min(n, 300)
    ind = np.concatenate([np.sort(g.choice(n, k, replace=False))
                          for k in lens]) if lens.sum() else np.zeros(0)
    ptr = np.concatenate([[0], np.cumsum(lens)])
    val = g.standard_normal(ind.size).astype(dtype)
    return sp.csr_matrix((val, ind.astype(np.int32), ptr.astype(np.int32)),
                         shape=(n, n))


def _check(A, x, y, t):
    eps = np.finfo(x.dtype).eps
    A64, x64 = A.astype(np.float64), x.astype(np.float64)
    want = A64 @ x64 + t * x64
    k = np.diff(A.indptr)[:, None]
    size = abs(A64) @ abs(x64) + abs(t * x64)
    assert np.all(np.abs(y - want) <= (k + 3) * eps * size + 1e-300)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("width", [32, 64, 128, 256, 512, 1024])
@pytest.mark.parametrize("n", [1, 7, 333, 3001])
def test_rows_product_at_every_width(cuda, dtype, width, n):
    import torch
    if dtype == np.float64 and width == 1024:
        pytest.skip("float64 blocks are at most 512 wide")
    A = _matrix(n, dtype, n + width)
    x = np.random.default_rng(5).standard_normal((n, width)).astype(dtype)
    for t in (0.0, 0.75):
        op = _DeviceOperator(A, t != 0.0, False, reorder=False, group_rows=0)
        y = op.dot(torch.from_numpy(x).cuda(), t=t).cpu().numpy()
        _check(A, x, y, t)


@pytest.mark.parametrize("dtype,width", [(np.float32, 32), (np.float32, 64),
                                         (np.float64, 32)])
def test_unaligned_buffers_are_still_taken(cuda, dtype, width):
    import torch
    n = 501
    A = _matrix(n, dtype, 3)
    op = _DeviceOperator(A, False, False, reorder=False, group_rows=0)
    x = np.random.default_rng(6).standard_normal((n, width)).astype(dtype)
    # one element (two at width 64, whose old kernel reads pairs) off
    off = 2 if width == 64 else 1
    xb = torch.zeros(n * width + off, dtype=torch.from_numpy(x).dtype,
                     device="cuda")
    yb = torch.zeros_like(xb)
    xb[off:] = torch.from_numpy(x.reshape(-1)).cuda()
    _lib.check(cuda.slq_operator_dot(
        op.handle, 0, 0.0, xb[off:].data_ptr(), yb[off:].data_ptr(), width,
        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    _check(A, x, yb[off:].cpu().numpy().reshape(n, width), 0.0)


def test_nonfinite_entries_reach_the_product(cuda):
    import torch
    n = 200
    A = sp.identity(n, dtype=np.float32, format="csr") * np.float32(2.0)
    x = np.ones((n, 64), np.float32)
    x[3, 5], x[4, 6] = np.inf, np.nan
    op = _DeviceOperator(A.tocsr(), False, False, reorder=False, group_rows=0)
    y = op.dot(torch.from_numpy(x).cuda()).cpu().numpy()
    assert np.isposinf(y[3, 5]) and np.isnan(y[4, 6])
    assert np.isfinite(y).sum() == y.size - 2


@pytest.mark.parametrize("width", [32, 256])
def test_samples_of_wide_blocks_match_narrow_ones(cuda, width):
    """The Krylov loop's product (scales, alpha partials in the epilogue) on
    wide float32 blocks against the 8-wide kernel on the same probes: single
    precision sums in the same order, so within rounding of the stored
    vectors (1e-6 of the estimate)."""
    A = _matrix(2000, np.float32, 9)
    A = (A @ A.T + 5.0 * sp.identity(2000)).tocsr().astype(np.float32)
    kw = dict(method="slq", gpu=True, return_info=True, min_num_samples=32,
              max_num_samples=width, error_rtol=0.0, lanczos_degree=20,
              orthogonalize=-1, seed=2)
    M = ib.Matrix(A, reorder=False, group_rows=0, blocks=False)
    _, wide = ib.logdet(M, block_size=width, **kw)
    _, narrow = ib.logdet(M, block_size=8, **dict(kw, max_num_samples=32))
    a = np.asarray(wide["convergence"]["samples"][:32], float)
    b = np.asarray(narrow["convergence"]["samples"][:32], float)
    assert np.max(np.abs(a - b) / np.abs(b)) < 1e-6


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("group_rows", [4, 8, 16])
@pytest.mark.parametrize("n", [3, 67, 1030])
def test_row_group_parts_equal_the_rows_product(cuda, dtype, group_rows, n):
    """Every row-group candidate (rows per warp x slices of the probes) gives
    the CSR product bit for bit: the same entries in the same order, the
    padding exact zeros -- at row counts that leave the last group ragged,
    unions around the four columns in flight, and every width."""
    import torch
    from imate_b200.batch import set_variant, tune_operator
    A = _matrix(n, dtype, n + group_rows)
    op = _DeviceOperator(A, True, True, reorder=False, aggregate=False,
                         group_rows=group_rows)
    for width in (32, 64, 128, 256):
        x = np.random.default_rng(width).standard_normal((n, width)) \
            .astype(dtype)
        X = torch.from_numpy(x).cuda()
        for tr in (False, True):
            for t in (0.0, 0.5):
                set_variant(op, width, 0, transpose=tr)
                base = op.dot(X, transpose=tr, t=t).cpu().numpy()
                _check((A.T if tr else A).tocsr(), x, base, t)
                cands, _ = tune_operator(op, width, transpose=tr, reps=1)
                for i, c in enumerate(cands):
                    if c["kind"] == "row-group":
                        set_variant(op, width, i, transpose=tr)
                        got = op.dot(X, transpose=tr, t=t).cpu().numpy()
                        assert np.array_equal(got, base), (width, tr, t, c)


def test_row_groups_with_unaligned_buffers_fall_back(cuda):
    import torch
    n, width = 400, 128
    A = _matrix(n, np.float32, 8)
    # (slq_operator_dot itself works in the stored row order: keep A's)
    op = _DeviceOperator(A, False, False, reorder=False, aggregate=False,
                         group_rows=16)
    x = np.random.default_rng(1).standard_normal((n, width)) \
        .astype(np.float32)
    xb = torch.zeros(n * width + 2, device="cuda")
    yb = torch.zeros_like(xb)
    xb[2:] = torch.from_numpy(x.reshape(-1)).cuda()
    _lib.check(cuda.slq_operator_dot(
        op.handle, 0, 0.0, xb[2:].data_ptr(), yb[2:].data_ptr(), width,
        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    _check(A, x, yb[2:].cpu().numpy().reshape(n, width), 0.0)
