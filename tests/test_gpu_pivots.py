"""The pivot kernel's groups at their edges (GPU): time lines of one step, one
group of four steps and one more; fewer than 32, exactly 32 and 33 (step, row)
pairs; row blocks and columns that end inside a chunk of 16 rows or a tile of
32 columns -- in every kernel family, against the FP64 oracle at the engine's
contract of 1e-9 relative."""
import importlib

import numpy as np
import pytest

from conftest import FIELDS

pytestmark = pytest.mark.gpu

wl = importlib.import_module("futhark-benchmarks_b200.workloads")


@pytest.mark.parametrize("numX,numY,numT", [(3, 3, 2), (32, 8, 5), (33, 11, 4), (31, 16, 3), (64, 32, 6), (65, 33, 2),
                                            (97, 47, 10), (300, 20, 6), (32, 256, 2), (256, 31, 9)])
def test_pivot_groups_vs_oracle(ctx, oracle, numX, numY, numT):
    c = wl.Calibration(5, numX, numY, numT, 0.033, 3.0, 0.22, 0.55, 0.45)
    want = oracle.main_f64(*[getattr(c, k) for k in FIELDS])
    got = ctx.main_f64(*[getattr(c, k) for k in FIELDS])
    assert np.max(np.abs(got - want) / np.maximum(np.abs(want), 1e-300)) <= 1e-9


def test_pivot_groups_of_several_calibrations(ctx, oracle):
    # groups of a plan: the prefix sums hold calibrations with no step at all,
    # and group counts that differ from calibration to calibration
    cs = [wl.Calibration(2, X, Y, T, 0.03, 4.0, 0.2, 0.5, 0.5)
          for X, Y, T in ((32, 32, 1), (64, 33, 6), (20, 7, 2), (32, 64, 5), (40, 5, 1), (128, 32, 3))]
    assert np.max(np.abs(ctx.batch(cs) / oracle.batch_f64(cs) - 1)) <= 1e-9
