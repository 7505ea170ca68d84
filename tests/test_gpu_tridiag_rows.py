"""The whole-row tridiagonal kernel where it can go wrong (GPU), bit for bit
against the CPU oracle: every alignment of the row length (accesses of one, two
and four elements, padded rows or not), lengths around the eight-element window,
partial last tiles, arrays off the 16-byte grid on either side, lengths where the
tile shrinks and where rows are read in place instead, and values outside the
range of its fast division -- zeros, negative zeros, tiny and huge ones,
infinities and NaN -- in some systems of a tile or all."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

wl = importlib.import_module("futhark-benchmarks_b200.workloads")
FORMS = [("seq", "seq"), ("par", "par4")]


def same(got, want):
    nan = np.isnan(want)
    return np.array_equal(nan, np.isnan(got)) and np.array_equal(got.view(np.int32)[~nan], want.view(np.int32)[~nan])


@pytest.mark.parametrize("rows,m", [(1, 1), (5, 2), (33, 7), (32, 8), (31, 9), (45, 15), (64, 16), (29, 17), (61, 18),
                                    (127, 20), (90, 24), (33, 31), (1000, 32), (77, 100), (41, 102), (300, 112),
                                    (25, 116), (20, 128), (23, 254), (9, 512), (11, 700), (6, 1599), (5, 1601),
                                    (7, 3000), (3, 4000), (150, 1800)])
@pytest.mark.parametrize("form,oform", FORMS)
def test_row_lengths_bit_exact(ctx, oracle, rows, m, form, oform):
    a, b, c, y = wl.tridiag_inputs(rows, m, seed=rows + m)
    assert same(ctx.tridag(a, b, c, y, form=form), oracle.tridag(a, b, c, y, form=oform))


@pytest.mark.parametrize("form,oform", FORMS)
@pytest.mark.parametrize("m", [23, 30, 64])
def test_values_out_of_the_fast_range(ctx, oracle, form, oform, m):
    rows = 96
    a, b, c, y = (v.copy() for v in wl.tridiag_inputs(rows, m, seed=m))
    special = [0.0, -0.0, 1e-30, -1e-38, 1e-44, 1e30, -3e38, np.inf, -np.inf, np.nan, 1e-13, 2e12]
    rng = np.random.default_rng(m)
    for r in range(40):  # tiles that mix ordinary systems and these
        for v in (a, b, c, y):
            if rng.random() < 0.4:
                v[r, rng.integers(m)] = special[rng.integers(len(special))]
    a[50], c[50] = 0.0, 0.0  # a diagonal system
    y[51] = -0.0
    y[52, 3:] = 0.0
    b[53], y[53] = 1e-20, 1e-25
    with np.errstate(all="ignore"):
        assert same(ctx.tridag(a, b, c, y, form=form), oracle.tridag(a, b, c, y, form=oform))


@pytest.mark.parametrize("off_in,off_out", [(1, 0), (0, 1), (2, 3)])
@pytest.mark.parametrize("m", [13, 64, 90])
def test_arrays_off_the_16_byte_grid(ctx, oracle, m, off_in, off_out):
    import torch
    rows = 70
    host = wl.tridiag_inputs(rows, m, seed=5)
    dev = []
    for v in host:
        t = torch.zeros(rows * m + 4, device="cuda:0")
        t[off_in:off_in + rows * m] = torch.from_numpy(v.ravel()).to("cuda:0")
        dev.append(t)
    out = torch.full((rows * m + 8,), 7.0, device="cuda:0")
    for form, oform in FORMS:
        torch.cuda.synchronize()
        ctx.tridag_device(form, rows, m, *[t[off_in:].data_ptr() for t in dev], out[off_out:].data_ptr())
        ctx.tridag_check()
        got = out.cpu().numpy()
        assert same(got[off_out:off_out + rows * m].reshape(rows, m), oracle.tridag(*host, form=oform))
        assert np.all(got[:off_out] == 7.0) and np.all(got[off_out + rows * m:] == 7.0)


@pytest.mark.parametrize("form,oform", FORMS)
def test_many_rows_of_long_systems_read_in_place(ctx, oracle, form, oform):
    rows, m = 148 * 16 * 4 + 4, 1700  # more rounds than the whole-row kernel takes beyond 1600 elements
    a, b, c, y = wl.tridiag_inputs(rows, m, seed=8)
    got = ctx.tridag(a, b, c, y, form=form)
    pick = np.r_[0:8, rows - 8:rows]
    assert same(got[pick], oracle.tridag(a[pick], b[pick], c[pick], y[pick], form=oform))
