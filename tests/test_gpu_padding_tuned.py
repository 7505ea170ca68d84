"""Padding that a tuned shape brings where memory is short (GPU): a call whose
padded tables do not fit is served without padding whether the padded shape is the
built-in choice or came out of the tuning table, and a server does so too when the
budget would cover the padded request but the blocks left in it do not hold its
tables."""
import ctypes
import importlib

import numpy as np
import pytest

from conftest import FIELDS

pytestmark = pytest.mark.gpu

wl = importlib.import_module("futhark-benchmarks_b200.workloads")
RTOL = 1e-9
LINE, PAIRS = 1, (3, 4)


def args(c):
    return [getattr(c, k) for k in FIELDS]


@pytest.fixture
def tuned_ctx(pkg):
    with pkg.Context("#0") as ctx:
        shape = [s for s in ctx.shape_candidates(200, 200) if s.family in PAIRS][0]
        ctx.tuning_set(200, 200, 0, shape)
        yield ctx


C200 = wl.Calibration(3, 200, 200, 161, 0.03, 5.0, 0.2, 0.6, 0.5)  # 76 MB of tables padded, 54 MB not


def test_no_allocation_call_under_a_tuned_shape(tuned_ctx, pkg, oracle):
    import torch
    lib = pkg.load_library()
    fn = lib.lvc_entry_main_f64_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p] + [ctypes.c_int32] * 4 + [ctypes.c_double] * 5
    assert 0 < lib.lvc_entry_main_f64_noalloc_bytes(tuned_ctx._ctx, 3, 200, 200, 161) <= 64 << 20
    out = torch.empty(3, dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    assert fn(tuned_ctx._ctx, ctypes.c_void_p(out.data_ptr()), *args(C200)) == 0, tuned_ctx._take_error()
    tuned_ctx.sync()
    assert np.max(np.abs(out.cpu().numpy() / oracle.main_f64(*args(C200)) - 1)) <= RTOL


def test_server_budget_under_a_tuned_shape(tuned_ctx, pkg, oracle):
    with pkg.Server(tuned_ctx, hbm_budget_bytes=60 << 20) as srv:
        got = srv.result(srv.submit(C200))
    assert np.max(np.abs(got / oracle.main_f64(*args(C200)) - 1)) <= RTOL


def test_plan_under_a_tuned_shape(pkg):
    import torch
    c = wl.Calibration(2, 33, 33, 60001, 0.03, 5.0, 0.2, 0.6, 0.5)  # 2.3 GB of tables padded, 0.7 GB not
    with pkg.Context("#0") as ctx:
        shapes = ctx.shape_candidates(33, 33)
        ctx.tuning_set(33, 33, 0, [s for s in shapes if s.family == LINE][0])
        want = ctx.batch([c])
    with pkg.Context("#0") as ctx:
        ctx.tuning_set(33, 33, 0, [s for s in shapes if s.family in PAIRS][0])
        ctx.batch([wl.Calibration(2, 64, 32, 9, 0.03, 5.0, 0.2, 0.6, 0.5)])
        free, _ = torch.cuda.mem_get_info()
        fill = torch.empty(free - (1536 << 20), dtype=torch.uint8, device="cuda")
        try:
            assert np.array_equal(ctx.batch([c]), want)
        finally:
            del fill
            torch.cuda.empty_cache()
