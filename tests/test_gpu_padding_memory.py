"""Padding where device memory is short (GPU): a plan and an entry point's call whose
padded tables do not fit are built without padding -- the same prices, bit for bit,
as the kernel for any sizes gives when it is asked for -- and one that does not fit
either way still fails as out of memory, after which the context works on."""
import importlib

import numpy as np
import pytest

from conftest import FIELDS

pytestmark = pytest.mark.gpu
wl = importlib.import_module("futhark-benchmarks_b200.workloads")
LINE = 1


def test_tables_that_fit_without_padding_only(pkg):
    import torch
    c = wl.Calibration(2, 33, 33, 60001, 0.03, 5.0, 0.2, 0.6, 0.5)  # 2.3 GB of tables padded, 0.7 GB not
    args = [getattr(c, k) for k in FIELDS]
    with pkg.Context("#0") as ctx:
        ctx.tuning_set(33, 33, 0, [s for s in ctx.shape_candidates(33, 33) if s.family == LINE][0])
        want = ctx.batch([c])
    with pkg.Context("#0") as ctx:
        small = wl.Calibration(2, 64, 32, 9, 0.03, 5.0, 0.2, 0.6, 0.5)
        before = ctx.batch([small])
        free, _ = torch.cuda.mem_get_info()
        fill = torch.empty(free - (1536 << 20), dtype=torch.uint8, device="cuda")
        try:
            assert np.array_equal(ctx.batch([c]), want)
            assert np.array_equal(ctx.main_f64(*args), want)
            with pytest.raises(Exception):
                ctx.batch([wl.Calibration(2, 33, 33, 600001, 0.03, 5.0, 0.2, 0.6, 0.5)])
        finally:
            del fill
            torch.cuda.empty_cache()
        assert np.array_equal(ctx.batch([small]), before)
