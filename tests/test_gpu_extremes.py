"""Krylov runs whose values leave FP32's range: blocks of 32 probes and more
(whose epilogue keeps off FP64 where it can) against the 8-wide kernel, which
computes in FP64 throughout, on the same probes.

Tolerance: the row sums and their order are the same and each product is the
double product rounded to FP32 up to ties, so coefficients differ by FP32
rounding at most: 1e-5 after six steps.  Powers of two as factors are exact."""

import contextlib

import numpy as np
import pytest
import scipy.sparse as sp

import imate_b200 as ib

pytestmark = pytest.mark.gpu


def _run(A, width, warns=False):
    """Samples, status bits and coefficients of eight probes."""
    M = ib.Matrix(A, reorder=False, group_rows=0, blocks=False)
    with pytest.warns() if warns else contextlib.nullcontext():
        _, info = ib.logdet(M, **_options(width))
    e = info["engine"]
    return [np.asarray(v[:8], float) for v in
            (info["convergence"]["samples"], e["probe_status"], e["alpha"],
             e["beta"])]


def _options(width):
    return dict(method="slq", gpu=True, return_info=True, min_num_samples=8,
                max_num_samples=8, error_rtol=0.0, lanczos_degree=6,
                orthogonalize=-1, seed=4,
                engine=ib.EngineOptions(block_size=width,
                                        return_coefficients=True))


def _matrix(n):
    g = np.random.default_rng(n)
    R = sp.random(n, n, density=8.0 / n, random_state=g, format="csr")
    return sp.csr_matrix(R + R.T + 12.0 * sp.identity(n)).astype(np.float32)


@pytest.mark.parametrize("width", [32, 128, 512])
@pytest.mark.parametrize("power", [0, -55, 55])
def test_scales_far_from_one(cuda, width, power):
    A = _matrix(1500) * np.float32(2.0**power)
    want, st8, _, _ = _run(A, 8)
    got, st, _, _ = _run(A, width)
    assert np.array_equal(st, st8) and np.all(st == 0)
    assert np.max(np.abs(got - want) / np.abs(want)) < 1e-5


@pytest.mark.parametrize("width", [32, 64, 256, 512, 1024])
@pytest.mark.parametrize("group_rows", [0, 4, 8, 16])
@pytest.mark.parametrize("mode", ["lanczos", "golub-kahn", "normal"])
def test_rows_far_below_the_others(cuda, width, group_rows, mode):
    # products below 2^-100: the threads of tiny rows take the FP64 products,
    # with alpha sums, norms or no sums (the first product of A^T A)
    n = 700
    A = sp.block_diag([_matrix(n), _matrix(300) * np.float32(2.0**-105)],
                      format="csr").astype(np.float32)
    def run(b, groups):
        from imate_b200.batch import set_variant, tune_operator
        extra = {}
        if mode == "normal":
            M = ib.GramAffineMatrixFunction(A)
            M.group_rows = groups
            extra["parameters"] = [1.0]
        else:
            M = ib.Matrix(A, reorder=False, group_rows=groups, blocks=False)
        if groups:
            op = M.get_device_operator(mode != "lanczos")
            cands, _ = tune_operator(op, b, reps=1)
            pick = [i for i, c in enumerate(cands) if c["kind"] == "row-group"]
            set_variant(op, b, pick[-1])
        _, info = ib.logdet(M, gram=mode == "golub-kahn", **extra,
                            **_options(b))
        e = info["engine"]
        return np.asarray(e["alpha"][:8], float), np.asarray(e["beta"][:8],
                                                             float)

    want = run(8, 0)
    for g, w in zip(run(width, group_rows), want):
        assert np.all(np.isfinite(w))
        assert np.max(np.abs(g - w)) < 1e-5 * np.max(np.abs(w))


@pytest.mark.parametrize("width", [32, 256])
@pytest.mark.parametrize("bad", [3.0e38, np.inf, np.nan])
def test_values_past_the_range_are_flagged_alike(cuda, width, bad):
    # a row that overflows (or holds a non-finite value) makes the next
    # Krylov vector, and with it the next alpha, non-finite
    A = _matrix(900).tolil()
    A[7, 8] = A[8, 7] = A[7, 9] = A[9, 7] = bad
    A = A.tocsr().astype(np.float32)
    want = _run(A, 8, warns=True)
    got = _run(A, width, warns=True)
    assert np.all(want[1].astype(int) & 1)
    assert np.array_equal(got[1].astype(int) & 1, want[1].astype(int) & 1)
    for g, w in zip(got, want):
        assert np.array_equal(np.isfinite(g), np.isfinite(w))
