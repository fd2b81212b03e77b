"""The six products of the dense operator's BF16 parts, where nothing but the
parts limits the result: one nonzero entry per row, full 24-bit mantissas.

The bound, in units of |a x|: a BF16 value has 8 significant bits, so |m| <=
2^-8 |v| and |l| <= 2^-16 |v|, and the products left out (m l, l m, l l) are
below 2^-23 + 2^-32.  The others are added smallest first, so that only the
last addition, of h h, is made at full size; the tensor core's FP32 addition is
taken to be off by at most 2^-22 of its result, the ones before it by 2^-22 of
2^-7.  2^-23 + 2^-22 (1 + 2^-6) < 2^-21 covers all."""

import numpy as np
import pytest

import imate_b200 as ib

BOUND = 2.0 ** -21
TERMS = ("lh", "mm", "hl", "mh", "hm", "hh")


def _bf16(v):
    """Round to nearest even to 8 significant bits (normal range)."""
    u = np.asarray(v, np.float32).view(np.uint32).astype(np.uint64)
    u = (u + 0x7fff + ((u >> 16) & 1)) & 0xffff0000
    return u.astype(np.uint32).view(np.float32)


def _parts(v):
    h = _bf16(v)
    m = _bf16(v - h)
    return {"h": h, "m": m, "l": _bf16(v - h - m)}


def _values(rng, n):
    """Full mantissas of magnitude 1 to 2, both signs, and among them those
    whose m, l or both are largest."""
    u = rng.integers(0, 2**23, n).astype(np.uint32)
    u[::5] = (u[::5] & 0x7f0000) | 0x7fff    # m and l near their largest
    u[1::5] = (u[1::5] & 0x7f0000) | 0x007f  # m zero, l largest
    u[2::5] = (u[2::5] & 0x7f0000) | 0x7f00  # m largest, l zero
    v = (u | 0x3f800000).view(np.float32)
    return v * rng.choice([-1, 1], n).astype(np.float32)


def _error(a, x, left_out=()):
    A, X = _parts(a), _parts(x)
    y = sum(A[t[0]].astype(np.float64) * X[t[1]] for t in TERMS
            if t not in left_out)
    want = a.astype(np.float64) * x
    return np.max(np.abs(y - want) / np.abs(want))


def test_the_bound_needs_every_product():
    rng = np.random.default_rng(0)
    a, x = _values(rng, 4000), _values(rng, 4000)
    assert np.array_equal(sum(p.astype(np.float64) for p in
                              _parts(a).values()), a)
    assert _error(a, x) < 2.0 ** -22
    for t in TERMS:
        assert _error(a, x, (t,)) > 8 * BOUND
    # a part taken for another one
    A, X = _parts(a), _parts(x)
    for t, s in (("lh", "mh"), ("hl", "hm"), ("mm", "ml")):
        off = np.abs(A[t[0]].astype(np.float64) * X[t[1]] -
                     A[s[0]].astype(np.float64) * X[s[1]])
        assert np.max(off / np.abs(a.astype(np.float64) * x)) > 8 * BOUND


@pytest.mark.gpu
@pytest.mark.parametrize("a_scale,x_scale", [(2.0**-100, 1.0), (1.0, 2.0**-100),
                                             (2.0**60, 2.0**-108),
                                             (2.0**-108, 2.0**60),
                                             (2.0**63, 2.0**62)])
def test_scales_far_from_one(cuda, a_scale, x_scale):
    # l is at least 2^-24 of a value: 2^-132, one of BF16's subnormals; sums of
    # the smallest products below 2^-126 may be lost, 3 * 2^-126 of 2^-100
    import torch
    rng = np.random.default_rng(3)
    a = _values(rng, 150)
    X = _values(rng, 150 * 40).reshape(150, 40)
    A = np.diag(a * np.float32(a_scale))
    op = ib.Matrix(A).get_device_operator()
    Y = op.dot(torch.from_numpy(X * np.float32(x_scale)).cuda()).cpu().numpy()
    want = a[:, None].astype(np.float64) * X * (a_scale * x_scale)
    assert np.max(np.abs(Y - want) / np.abs(want)) <= BOUND


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,width", [
    (130, 1, 48), (300, 200, 16), (129, 97, 256), (9700, 64, 33),
    (70, 2100, 300)])
@pytest.mark.parametrize("transpose", [False, True])
def test_one_entry_per_row(cuda, rows, cols, width, transpose):
    import torch
    rng = np.random.default_rng(rows + cols + width)
    out, inner = (cols, rows) if transpose else (rows, cols)
    a = _values(rng, out)
    at = rng.integers(0, inner, out)
    S = np.zeros((out, inner), np.float32)
    S[np.arange(out), at] = a
    X = _values(rng, inner * width).reshape(inner, width)
    op = ib.Matrix(np.ascontiguousarray(S.T if transpose else S)) \
        .get_device_operator(need_transpose=True)
    assert getattr(op, "dense", False)
    Y = op.dot(torch.from_numpy(X).cuda(), transpose=transpose).cpu().numpy()
    want = a[:, None].astype(np.float64) * X[at]
    assert np.max(np.abs(Y - want) / np.abs(want)) <= BOUND
