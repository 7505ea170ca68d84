"""The tke step where its fast divisions can go wrong (GPU), bit for bit against
the CPU oracle: depths around the column kernel's chunk of four levels, plane
sizes around the advection kernel's tiles, and fields, grid spacings and
velocities outside the range of the fast division, in some columns or all."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = importlib.import_module("futhark-benchmarks_b200.workloads")
tke_mod = importlib.import_module("futhark-benchmarks_b200.tke")


@pytest.fixture(scope="module")
def tctx():
    with tke_mod.TkeContext() as c:
        yield c


def check(tctx, oracle, ins):
    with np.errstate(all="ignore"):
        want = oracle.tke(*ins)
    for g, w in zip(tctx.main(*ins), want):
        nan = np.isnan(w)
        assert np.array_equal(nan, np.isnan(g))
        assert np.array_equal(g.view(np.int32)[~nan], w.view(np.int32)[~nan])


@pytest.mark.parametrize("dims", [(5, 5, 2), (6, 7, 3), (9, 12, 4), (7, 40, 5), (12, 9, 8), (6, 10, 31), (5, 19, 33),
                                  (33, 6, 64)])
def test_depths_and_tiles(tctx, oracle, dims):
    check(tctx, oracle, W.tke_inputs(*dims, seed=sum(dims), wet=True))


@pytest.mark.parametrize("name", ["tketau", "utau", "vtau", "wtau", "kappaM", "mxl", "forc", "maskW"])
@pytest.mark.parametrize("value", [0.0, -0.0, 1e-30, 1e-40, -3e19, 1e35, np.inf, np.nan])
def test_field_values_out_of_range(tctx, oracle, name, value):
    ins = list(W.tke_inputs(14, 12, 9, seed=3, wet=True))
    v = np.array(ins[tke_mod.INPUT_NAMES.index(name)])
    rng = np.random.default_rng(5)
    v[rng.random(v.shape) < 0.02] = value
    v[7] = value  # and a whole slice of columns
    ins[tke_mod.INPUT_NAMES.index(name)] = v
    check(tctx, oracle, ins)


@pytest.mark.parametrize("name", ["dxt", "dyt", "dzt", "dzw", "cost", "cosu"])
@pytest.mark.parametrize("value", [1e-7, 1e-13, 3e6, 1e13, -0.5])
def test_grid_spacings_out_of_range(tctx, oracle, name, value):
    for where in (slice(4, 5), slice(None)):
        ins = list(W.tke_inputs(14, 12, 9, seed=4, wet=True))
        v = np.array(ins[tke_mod.INPUT_NAMES.index(name)])
        v[where] = value
        ins[tke_mod.INPUT_NAMES.index(name)] = v
        check(tctx, oracle, ins)


@pytest.mark.parametrize("scale", [1e-12, 1e-25, 1e-36, 1e12])
def test_states_of_other_scales(tctx, oracle, scale):
    # tiny differences of the state: dividends below the range of the fast quotient
    ins = list(W.tke_inputs(12, 14, 10, seed=6, wet=True))
    for n in ("tketau", "tketaup1", "utau", "vtau", "wtau", "forc", "forc_tke_surface"):
        k = tke_mod.INPUT_NAMES.index(n)
        ins[k] = (ins[k] * np.float32(scale)).astype(np.float32)
    check(tctx, oracle, ins)
