"""Contract 2 with its tail Gaussians queued per warp (GPU), against the CPU oracle --
bit for bit in path order, to 1e-6 in the default order, whose f64 sums differ in
their grouping: path counts around a warp, and around the ones from which the 1184
CTAs of 128 threads that 148 SMs get take one, two and three paths per thread, some
lanes of a warp one more than others."""
import importlib

import numpy as np
import pytest

from conftest import golden_npz

pytestmark = pytest.mark.gpu
THREADS = 8 * 148 * 128


@pytest.fixture(scope="module")
def contexts():
    op = importlib.import_module("futhark-benchmarks_b200.op")
    with op.OpContext() as seq, op.OpContext() as f64:
        seq.set_reduction_order(seq.ORDER_SEQUENTIAL_F32)
        yield seq, f64


@pytest.mark.parametrize("paths,models", [
    (1, 1), (31, 2), (33, 5), (THREADS - 1, 1), (THREADS, 1), (THREADS + 1, 2), (2 * THREADS + 777, 1),
])
def test_against_oracle(contexts, oracle, paths, models):
    z = golden_npz("optionpricing_medium")
    ins = [z[f"in{i:02d}"] for i in range(11)]
    ins[1] = np.int32(paths)
    rng = np.random.default_rng(paths)
    for k in range(3, 9):
        ins[k] = np.repeat(ins[k], models, axis=0)
    ins[6] = (ins[6] * rng.uniform(0.9, 1.2, ins[6].shape)).astype(np.float32)
    seq, f64 = contexts
    assert np.array_equal(seq.main(*ins), oracle.option_pricing(*ins, order="sequential_f32"))
    assert np.allclose(f64.main(*ins), oracle.option_pricing(*ins), rtol=1e-6, atol=0)
