"""Arrays of the generated API whose sizes do not divide the device pool's 256 MB
chunks (GPU): one may not be carved across two chunks that happen to be
neighbours, since a copy cannot span two allocations."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

wl = importlib.import_module("futhark-benchmarks_b200.workloads")


def test_arrays_past_a_chunk_copy_back(pkg, oracle):
    a, b, c, y = wl.tridiag_inputs(9476, 1700, seed=8)  # 64.4 MB each: the fourth array opens a second chunk
    with pkg.Context("#0") as ctx:
        for _ in range(3):
            got = ctx.tridag(a, b, c, y, form="seq")
    assert np.array_equal(got[:4], oracle.tridag(a[:4], b[:4], c[:4], y[:4], form="seq"))
