"""A server request that its HBM budget covers while the plans kept idle split the
room left (GPU): they are released and the request is served, instead of failing as
out of memory."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

wl = importlib.import_module("futhark-benchmarks_b200.workloads")


def request(numT):  # 36.5 KiB of tables a step
    return wl.Calibration(2, 33, 33, numT, 0.03, 5.0, 0.2, 0.6, 0.5)


def test_request_larger_than_the_gaps_between_idle_plans(ctx, pkg):
    # plans of 91 MiB each at the start of 300; the third needs 146: room once the first
    # is released, but in two pieces of 91 and 117
    sizes = (2500, 2501, 4000)
    want = [ctx.batch([request(T)]) for T in sizes]
    with pkg.Server(ctx, hbm_budget_bytes=300 << 20) as srv:
        for T, w in zip(sizes, want):
            assert np.array_equal(srv.result(srv.submit(request(T))), w)
        tickets = [srv.submit(request(T)) for T in sizes]
        for t, w in zip(tickets, want):
            assert np.array_equal(srv.result(t), w)
        assert srv.stats()["failed"] == 0
