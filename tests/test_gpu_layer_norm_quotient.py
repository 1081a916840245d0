"""The quotient of the 16-bit path's layer norm is the correctly rounded one.

With ln0's weight 0 every embedded row is ln0's bias, which the test chooses: whole numbers of sum 0 times a power of
two, so mean and variance are exact in any order and the state's first row is the quotient alone."""
import numpy as np
import pytest
import torch

from rwkvstic_b200.dense_model import B200DenseRWKV

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("embed,T", [(1024, 1), (1024, 3), (4096, 1), (8192, 2)])      # one and two groups of inputs per thread
def test_the_quotient_is_the_correctly_rounded_one(embed, T):
    model = B200DenseRWKV.synthetic(1, embed, vocab=64, seed=1, dtype=torch.float16, device=DEV, use_graph=False)
    model.t["blocks.0.ln0.weight"].zero_()
    tokens = torch.arange(T).reshape(1, T)
    rng = np.random.default_rng(embed + T)
    for i in range(120):
        half = rng.integers(-60, 61, embed // 2)                   # sum of squares at most 8192 * 3600 / 2 < 2^24
        row = np.concatenate([half, -half]).astype(np.float32)
        rng.shuffle(row)
        row *= np.float32(2.0) ** rng.integers(-40, 41)
        var = np.float32(np.sum(row.astype(np.float64) ** 2)) / np.float32(embed)
        want = row / np.sqrt(var + np.float32(1e-5))
        model.t["blocks.0.ln0.bias"].copy_(torch.from_numpy(row))
        state = model.empty_batch_state(1)
        model.forward_rows(tokens, state)
        assert np.array_equal(state[0, 0, 0].cpu().numpy(), want), i
    model.check_status()


def test_a_spread_beyond_the_range_gives_zeros():
    """The squares overflow, the deviation is infinite, and the quotient by it is 0, not NaN."""
    model = B200DenseRWKV.synthetic(1, 1024, vocab=64, seed=1, dtype=torch.float16, device=DEV, use_graph=False)
    model.t["blocks.0.ln0.weight"].zero_()
    row = torch.ones(1024)
    row[::2] = -1.0
    model.t["blocks.0.ln0.bias"].copy_(row * 1e25)
    state = model.empty_batch_state(1)
    model.forward_rows(torch.zeros(1, 2, dtype=torch.int64), state)
    assert float(state[0, 0, 0].abs().max()) == 0.0
