"""The tall paired kernel (GPU): every column width, odd and even cluster sizes,
grids one off its tiles on either side, one and several steps, against the FP64
oracle (1e-9, the contract's tolerance), and at the strikes where the built-in
choice takes it, several items per CTA and all strikes the same as alone."""
import importlib

import numpy as np
import pytest

from conftest import FIELDS

pytestmark = pytest.mark.gpu

wl = importlib.import_module("futhark-benchmarks_b200.workloads")
RTOL = 1e-9
LINE_TALL = 5
SIZES = [(64, 256), (128, 128), (256, 64), (63, 255), (65, 129), (127, 257), (193, 33), (255, 65), (256, 128),
         (200, 190), (64, 700), (128, 512), (256, 256), (240, 300), (250, 512), (16, 40)]


def args(c):
    return [getattr(c, k) for k in FIELDS]


@pytest.mark.parametrize("X,Y", SIZES, ids=[f"{x}x{y}" for x, y in SIZES])
def test_tall_vs_oracle(ctx, oracle, X, Y):
    tall = [s for s in ctx.shape_candidates(X, Y) if s.family == LINE_TALL]
    assert len(tall) == 1
    try:
        ctx.tuning_set(X, Y, 0, tall[0])
        for numT in (1, 2, 6):
            c = wl.Calibration(5, X, Y, numT, 0.034, 4.0, 0.23, 0.55, 0.45)
            want = oracle.main_f64(*args(c))
            got = ctx.batch([c])
            assert np.max(np.abs(got / want - 1)) <= RTOL
            many = ctx.batch([wl.Calibration(301, *args(c)[1:])])  # more strikes than clusters on the chip
            assert np.array_equal(many[:5], got)
    finally:
        ctx.tuning_set(X, Y, 0, None)


def test_not_offered_beyond_its_grids(ctx):
    for X, Y, prec in ((257, 64, 0), (192, 64, 0), (256, 520, 0), (256, 256, 1)):
        assert not [s for s in ctx.shape_candidates(X, Y, prec) if s.family == LINE_TALL]


def test_built_in_choice(ctx, oracle):
    assert ctx.tuning_get(128, 256).shape.family == LINE_TALL
    assert ctx.tuning_get(128, 128).shape.family != LINE_TALL
    assert ctx.tuning_get(256, 256).shape.family != LINE_TALL  # in batches
    for outer in (6, 64):  # the paired kernel, the tall one
        c = wl.Calibration(outer, 256, 256, 4, 0.03, 5.0, 0.2, 0.6, 0.5)
        assert np.max(np.abs(ctx.main_f64(*args(c))[:6] / oracle.main_f64(6, *args(c)[1:]) - 1)) <= RTOL
