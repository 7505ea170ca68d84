"""Tridiagonal solves whose right-hand side is a few elements, tiny or subnormal, so that
what the recurrences carry goes through all magnitudes down to zero (GPU): row lengths
around the eight-element window at every access width, bit for bit against the CPU
oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(got, want):
    nan = np.isnan(want)
    return np.array_equal(nan, np.isnan(got)) and np.array_equal(got.view(np.int32)[~nan], want.view(np.int32)[~nan])


@pytest.mark.parametrize("form,oform", [("seq", "seq"), ("par", "par4")])
@pytest.mark.parametrize("m", [1, 2, 5, 7, 8, 9, 15, 16, 17, 24, 30, 33, 64, 100, 115, 130])
def test_fading_right_hand_sides(ctx, oracle, m, form, oform):
    rows = 130
    rng = np.random.default_rng(m)
    u = lambda: (rng.random((rows, m)) + 0.3).astype(np.float32)  # noqa: E731
    lower, upper, y = u(), u(), u()
    weak = np.float32(0.01) ** rng.integers(0, 3, (rows, 1)).astype(np.float32)
    a, b, c = -lower * weak, np.float32(1.0) + lower + upper, -upper * weak
    kind = np.arange(rows) % 5
    y[kind == 0, m // 3 + 1:] = 0.0          # a source at the start
    y[kind == 1] = 0.0
    y[kind == 1, m // 2] = -1.0              # one element
    y[kind == 2] *= np.float32(1e-30)
    y[kind == 3] *= np.float32(1e-42)        # subnormal
    assert same(ctx.tridag(a, b, c, y, form=form), oracle.tridag(a, b, c, y, form=oform))
