"""tridagPar where the scan of the pivots overflows while everything that the fast
divisions see stays in their range (GPU): b'_i is then infinite, and at the last
element the solution is finite.  Bit for bit against the CPU oracle, alone and in a
tile of ordinary systems, at every access width of the whole-row kernel."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

wl = importlib.import_module("futhark-benchmarks_b200.workloads")


def same(got, want):
    nan = np.isnan(want)
    return np.array_equal(nan, np.isnan(got)) and np.array_equal(got.view(np.int32)[~nan], want.view(np.int32)[~nan])


def solve(ctx, oracle, ins):
    with np.errstate(all="ignore"):
        want = oracle.tridag(*ins, form="par4")
    assert same(ctx.tridag(*ins, form="par"), want)
    return want


def test_overflow_in_a_system_of_two(ctx, oracle):
    f = lambda *v: np.array([v], np.float32)  # noqa: E731
    want = solve(ctx, oracle, (f(0, 1e14), f(1, 1e-11), f(1e14, 0), f(1, 1)))
    assert np.array_equal(want, f(1, 0))


@pytest.mark.parametrize("m", [5, 6, 16, 17, 24, 115])
def test_overflow_at_the_last_element(ctx, oracle, m):
    rows = 70
    rng = np.random.default_rng(m)
    u = lambda: (rng.random((rows, m)) + 0.3).astype(np.float32)  # noqa: E731
    lower, upper, y = u(), u(), u()
    a, b, c = -lower, np.float32(1.0) + lower + upper, upper  # all terms of the scan positive: no inf - inf
    hit = rng.random(rows) < 0.3
    hit[[0, 41]] = True
    a[hit, m - 1] = -np.ldexp(rng.uniform(0.5, 1, hit.sum()), 79).astype(np.float32)
    c[hit, m - 2] = np.float32(2.0**60)
    want = solve(ctx, oracle, (a, b, c, y))
    assert np.all(np.isfinite(want))


def test_overflow_inside_and_nan_inputs(ctx, oracle):
    rows, m = 64, 20
    a, b, c, y = (v.copy() for v in wl.tridiag_inputs(rows, m, seed=11))
    for r in range(rows):
        i = 1 + r % (m - 1)
        a[r, i], c[r, i - 1] = -(2.0**78), 2.0**55
    b[5, 3] = y[9, 0] = a[17, 18] = np.nan
    solve(ctx, oracle, (a, b, c, y))


@pytest.mark.parametrize("form,oform", [("seq", "seq"), ("par", "par4")])
@pytest.mark.parametrize("m", [7, 20, 115])
def test_matrices_of_any_scale(ctx, oracle, m, form, oform):
    rows = 64
    a, b, c, y = (v.copy() for v in wl.tridiag_inputs(rows, m, seed=m))
    for r in range(rows):  # pivots from below the normal floats to their upper end
        s = np.float32(2.0 ** (-128 + 4 * r))
        a[r], b[r], c[r] = a[r] * s, b[r] * s, c[r] * s
    with np.errstate(all="ignore"):
        assert same(ctx.tridag(a, b, c, y, form=form), oracle.tridag(a, b, c, y, form=oform))
