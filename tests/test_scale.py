"""An FP32 value times an FP64 probe scale is the double product rounded to
FP32 over the whole range of both types, non-finite values included.

The FP32 pair carries the product to 2^-48 of itself, so the result may differ
from the double product's only where that lies within 2^-24 of an FP32 spacing
of a tie; the fraction of random products there is 2^-23, and the comparison
allows a difference of one spacing in 1e-6 of them."""

import ctypes

import numpy as np
import pytest

import native


@pytest.fixture(scope="module")
def scale(tmp_path_factory):
    lib = native.load("scale", tmp_path_factory.mktemp("scale"))

    def run(x, s):
        x = np.ascontiguousarray(x, np.float32)
        s = np.ascontiguousarray(s, np.float64)
        y, b = np.empty_like(x), np.empty_like(s)
        w, n = np.empty(x.size, np.int32), np.empty_like(x)
        lib.scale(x.size, *[ctypes.c_void_p(v.ctypes.data)
                            for v in (x, s, y, w, b, n)])
        bad = ~np.isfinite(x)
        assert np.all(np.isnan(n[bad]))
        assert np.array_equal(n[~bad], y[~bad], equal_nan=True)
        return y, w, b
    return run


def _check(x, s, y):
    with np.errstate(all="ignore"):
        want = (x.astype(np.float64) * s).astype(np.float32)
    same = (y == want) | (np.isnan(y) & np.isnan(want))
    off = ~same
    assert np.count_nonzero(off) <= 1e-6 * x.size
    assert np.all(np.abs(y[off] - want[off]) <= np.spacing(np.abs(want[off])))


@pytest.mark.parametrize("seed", [0, 1])
def test_every_exponent_of_value_and_scale(scale, seed):
    g = np.random.default_rng(seed)
    n = 3000000
    x = np.ldexp(1.0 + g.random(n), g.integers(-150, 128, n)) \
        .astype(np.float32) * g.choice([-1, 1], n).astype(np.float32)
    s = np.ldexp(1.0 + g.random(n), g.integers(-200, 160, n))
    y, wide, back = scale(x, s)
    _check(x, s, y)
    assert np.array_equal(back, x.astype(np.float64))
    # the pair serves whatever is in its range
    p = np.abs(x.astype(np.float64) * s)
    fits = (s >= 2.0**-100) & (s <= 2.0**126) & (p > 2.0**-99) & \
        (p < 2.0**125)
    assert not np.any(wide[fits])


def test_edges(scale):
    x = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 3.4028235e38,
                  1e-45, -1e-45, 1.1754944e-38, 1.7e38], np.float32)
    s = np.array([0.0, 1.0, 0.1, 2.0**-100, 2.0**100, np.nextafter(2.0**-100, 0),
                  np.nextafter(2.0**100, np.inf), 1e-300, 1e300, 2.0**149,
                  np.inf, np.nan, 1.0 - 2.0**-50, 1.0 + 2.0**-52])
    X, S = [v.ravel() for v in np.meshgrid(x, s)]
    y, _, _ = scale(X, S)
    with np.errstate(all="ignore"):
        want = (X.astype(np.float64) * S).astype(np.float32)
    assert np.array_equal(y, want, equal_nan=True)


def test_ordinary_values_and_zeros_need_no_second_product(scale):
    g = np.random.default_rng(2)
    x = g.standard_normal(100000).astype(np.float32)
    x[::3] = 0.0
    _, wide, _ = scale(x, np.full(x.size, 0.0123456789))
    assert not np.any(wide)


def test_a_stopped_probe_needs_no_second_product(scale):
    # its scale is zero, its vector is not
    x = np.random.default_rng(3).standard_normal(1000).astype(np.float32)
    y, wide, _ = scale(x, np.zeros(x.size))
    assert not np.any(wide) and not np.any(y)
