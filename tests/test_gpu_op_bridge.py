"""Contract 3's two kernels (GPU), bit for bit against the CPU oracle in path order
and to 1e-6 in the default order: bridges filled in place 32 paths at a time --
path counts around a block, several models, directions of few bits -- and index
patterns that are no bridge (a date filled twice, never, or read before it is
filled), which the warp-per-path kernel prices."""
import importlib

import numpy as np
import pytest

from conftest import golden_npz

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def contexts():
    op = importlib.import_module("futhark-benchmarks_b200.op")
    with op.OpContext() as seq, op.OpContext() as f64:
        seq.set_reduction_order(seq.ORDER_SEQUENTIAL_F32)
        yield seq, f64


def daily(paths, models=1, seed=0):
    z = golden_npz("optionpricing_large")
    ins = [z[f"in{i:02d}"] for i in range(11)]
    ins[1] = np.int32(paths)
    rng = np.random.default_rng(seed)
    for k in range(3, 9):
        ins[k] = np.repeat(ins[k], models, axis=0)
    ins[6] = (ins[6] * rng.uniform(0.7, 1.1, ins[6].shape)).astype(np.float32)
    ins[4] = (ins[4] * rng.uniform(0.1, 1.2, ins[4].shape)).astype(np.float32)
    return ins


def check(contexts, oracle, ins):
    seq, f64 = contexts
    assert np.array_equal(seq.main(*ins), oracle.option_pricing(*ins, order="sequential_f32"))
    assert np.allclose(f64.main(*ins), oracle.option_pricing(*ins), rtol=1e-6, atol=0)


@pytest.mark.parametrize("paths,models", [(1, 1), (30, 1), (31, 1), (32, 2), (33, 1), (63, 5), (64, 1), (4735, 1),
                                          (4736, 3)])
def test_path_counts(contexts, oracle, paths, models):
    check(contexts, oracle, daily(paths, models, seed=paths))


@pytest.mark.parametrize("bits", [3, 5, 17, 31])
def test_direction_bits(contexts, oracle, bits):
    ins = daily(200)
    dirs = np.random.default_rng(bits).integers(1, 1 << min(bits, 30), (1101, bits))
    ins[2] = dirs.astype(np.int32)
    check(contexts, oracle, ins)


@pytest.mark.parametrize("kind", ["twice", "early", "self", "left", "shuffled"])
def test_other_index_patterns(contexts, oracle, kind):
    ins = daily(70)
    ind = np.array(ins[9])
    if kind == "twice":
        ind[0, 200] = ind[0, 100]
    elif kind == "early":  # a step reads a date that a later one fills
        ind[2, 5] = ind[0, 300]
    elif kind == "self":
        ind[2, 50] = ind[0, 50]
    elif kind == "left":
        ind[1, 40] = ind[0, 41]
    else:  # a bridge still: steps in another order that fills before it reads
        order = np.r_[0, 1 + np.argsort([max(1, int(i)) for i in np.floor(np.log2(np.arange(1, 367)))], kind="stable")]
        ind = ind[:, order]
        ins[10] = np.array(ins[10])[:, order]
    ins[9] = np.ascontiguousarray(ind.astype(np.int32))
    check(contexts, oracle, ins)
