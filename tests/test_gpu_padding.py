"""Grids padded to whole tiles for the paired kernel (GPU): sizes one off a tile
on either side, odd cluster sizes, every thread count the padding brings, both
precisions, against the FP64 oracle and the kernel for any sizes at the
contracts' tolerances (1e-9; 1e-4 on prices above 1e-3 of the largest with FP32
state).  And what padding must not change: a call whose padded tables do not fit
the static scratch or a server's budget is served without padding."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import FIELDS

pytestmark = pytest.mark.gpu

wl = importlib.import_module("futhark-benchmarks_b200.workloads")
F64_RTOL, F32S_RTOL = 1e-9, 1e-4
LINE_PAIR, LINE_PAIR1, LINE_TALL, LINE = 3, 4, 5, 1
SIZES = [(31, 31), (33, 32), (63, 65), (64, 96), (65, 95), (96, 192), (97, 33), (129, 160), (160, 129), (192, 32),
         (193, 97), (255, 225), (70, 250), (4, 255), (256, 33)]


def args(c):
    return [getattr(c, k) for k in FIELDS]


@pytest.mark.parametrize("X,Y", SIZES, ids=[f"{x}x{y}" for x, y in SIZES])
def test_padded_grid_vs_oracle_and_unpadded(ctx, oracle, X, Y):
    c = wl.Calibration(6, X, Y, 7, 0.034, 4.0, 0.23, 0.55, 0.45)
    want = oracle.main_f64(*args(c))
    assert ctx.tuning_get(X, Y).shape.family in (LINE_PAIR, LINE_PAIR1, LINE_TALL)
    got = ctx.batch([c])
    assert np.max(np.abs(got / want - 1)) <= F64_RTOL
    # alone, with strikes that fill the chip or do not: other splits
    assert np.max(np.abs(ctx.main_f64(*args(c)) / want - 1)) <= F64_RTOL
    many = wl.Calibration(300, *args(c)[1:])
    assert np.max(np.abs(ctx.main_f64(*args(many))[:6] / want - 1)) <= F64_RTOL
    half = ctx.batch([c], precision=1)
    big = want > 1e-3 * np.max(want)
    assert np.max(np.abs(half[big] / want[big] - 1)) <= F32S_RTOL
    assert np.max(np.abs(half[~big] - want[~big]), initial=0.0) <= 1e-7
    line = [s for s in ctx.shape_candidates(X, Y) if s.family == LINE]
    try:
        for s in line[:1]:
            ctx.tuning_set(X, Y, 0, s)
            assert np.max(np.abs(got / ctx.batch([c]) - 1)) <= F64_RTOL
    finally:
        ctx.tuning_set(X, Y, 0, None)


def test_no_allocation_call_that_fits_without_padding_only(pkg, oracle):
    import torch
    c = wl.Calibration(3, 200, 200, 161, 0.03, 5.0, 0.2, 0.6, 0.5)  # 76 MB of tables padded, 54 MB not
    with pkg.Context("#0") as ctx:
        lib = pkg.load_library()
        fn = lib.lvc_entry_main_f64_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p] + [ctypes.c_int32] * 4 + [ctypes.c_double] * 5
        assert 0 < lib.lvc_entry_main_f64_noalloc_bytes(ctx._ctx, 3, 200, 200, 161) <= 64 << 20
        out = torch.empty(3, dtype=torch.float64, device="cuda:0")
        torch.cuda.synchronize()
        assert fn(ctx._ctx, ctypes.c_void_p(out.data_ptr()), *args(c)) == 0, ctx._take_error()
        ctx.sync()
        assert np.max(np.abs(out.cpu().numpy() / oracle.main_f64(*args(c)) - 1)) <= F64_RTOL


def test_server_budget_that_fits_without_padding_only(ctx, pkg, oracle):
    c = wl.Calibration(3, 200, 200, 161, 0.03, 5.0, 0.2, 0.6, 0.5)
    small = wl.Calibration(3, 64, 32, 9, 0.03, 5.0, 0.2, 0.6, 0.5)
    with pkg.Server(ctx, hbm_budget_bytes=60 << 20) as srv:
        tickets = [srv.submit(k) for k in (small, c, small, c)]
        got = [srv.result(t) for t in tickets]
    assert np.max(np.abs(got[1] / oracle.main_f64(*args(c)) - 1)) <= F64_RTOL
    assert np.array_equal(got[1], got[3]) and np.array_equal(got[0], got[2])
