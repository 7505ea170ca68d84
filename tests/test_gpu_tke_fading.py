"""Columns in which the energy fades out (GPU): the state and the forcing are zero, tiny
or subnormal above the sea floor, so that what the recurrences carry up goes through all
magnitudes down to zero -- bit for bit against the CPU oracle, where a lane moves four
levels at a time and where it does not."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = importlib.import_module("futhark-benchmarks_b200.workloads")
tke_mod = importlib.import_module("futhark-benchmarks_b200.tke")


@pytest.mark.parametrize("Z", [8, 21, 40, 64])
@pytest.mark.parametrize("diffusion", [1e-6, 1e-2, 1.0])
@pytest.mark.parametrize("above", [0.0, 1e-30, 1e-42])
def test_energy_at_the_sea_floor_only(oracle, Z, diffusion, above):
    ins = list(W.tke_inputs(9, 11, Z, seed=Z, wet=True))
    at = {n: k for k, n in enumerate(tke_mod.INPUT_NAMES)}
    rng = np.random.default_rng(Z)
    for n in ("tketau", "forc"):
        v = np.abs(ins[at[n]])
        v[:, :, 3:] = above * rng.random((9, 11, Z - 3))
        ins[at[n]] = v.astype(np.float32)
    ins[at["kappaM"]] = (ins[at["kappaM"]] * np.float32(diffusion)).astype(np.float32)
    ins[at["kbot"]] = rng.integers(0, 3, (9, 11)).astype(np.int32)
    ins[at["forc_tke_surface"]] = np.zeros((9, 11), np.float32)
    with np.errstate(all="ignore"):
        want = oracle.tke(*ins)
    with tke_mod.TkeContext() as tctx:
        for g, w in zip(tctx.main(*ins), want):
            assert np.array_equal(g.view(np.int32), w.view(np.int32))
