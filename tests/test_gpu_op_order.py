"""The sum over paths in path order (f32 running sum), bit for bit against the
oracle, where its blocks can go wrong (GPU): path counts at the edges of a
256-payoff block and of one step of the composition (4096 blocks), a second
window of models, and payoffs that are mostly or all zero -- runs of zero
blocks, and blocks whose exponent the mean payoff does not predict."""
import importlib

import numpy as np
import pytest

from conftest import golden_npz

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def seq_ctx():
    op = importlib.import_module("futhark-benchmarks_b200.op")
    with op.OpContext() as c:
        c.set_reduction_order(c.ORDER_SEQUENTIAL_F32)
        yield c


def european(paths, starts):
    """The small dataset's European call, one model per start price."""
    z = golden_npz("optionpricing_small")
    ins = [z[f"in{i:02d}"] for i in range(11)]
    ins[1] = np.int32(paths)
    for k in (3, 4, 5, 7, 8):
        ins[k] = np.repeat(ins[k], len(starts), axis=0)
    ins[6] = np.array(starts, np.float32)[:, None]
    return ins


@pytest.mark.parametrize("paths,starts", [
    (255, [3758.05]), (256, [3758.05]), (257, [3758.05, 4100.0]), (1024 * 4 * 256, [3758.05]),
    (1024 * 4 * 256 + 1, [3758.05]), (300000, [3700.0, 3800.0, 3900.0, 4000.0, 4100.0]),
    (1 << 20, [2000.0, 2200.0, 2400.0, 2600.0]),  # a payoff in a thousand to a hundred thousand paths
    (5000, [500.0]),  # none: all blocks zero
])
def test_path_order_sum_bit_for_bit(seq_ctx, oracle, paths, starts):
    ins = european(paths, starts)
    assert np.array_equal(seq_ctx.main(*ins), oracle.option_pricing(*ins, order="sequential_f32"))
