"""The WKV scan of the prompt path where its chunks and its arithmetic can go wrong, against the one-row path (one
token at a time, the same fp32 recurrence step by step)."""
import pytest
import torch

from rwkvstic_b200.model import B200RWKV
from rwkvstic_b200.synth import synth_checkpoint, synth_tokens

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
V = 257


def compare(ck, state, B, T):
    model = B200RWKV.from_checkpoint(ck, device=DEV, use_graph=False)
    model.rows_threshold = 1 << 30              # forward() takes the one-row path whatever the length
    tokens = synth_tokens(B * T, seed=9, vocab=V).reshape(B, T)
    rows, one = state(model, B), state(model, B)
    lg_rows, _ = model.forward_batch(tokens, rows, rows=True)
    lg_one, _ = model.forward_batch(tokens, one, rows=False)
    assert bool(torch.isfinite(lg_one).all())
    # fp32 layer norms and scans summed in another order, as in test_rows_path_agrees_with_one_row_path
    assert float((lg_rows - lg_one).abs().max()) < 2e-4
    assert torch.allclose(rows[:, :, :4], one[:, :, :4], rtol=1e-4, atol=1e-4)
    model.check_status()


@pytest.mark.parametrize("T", [2, 5, 40])
def test_a_state_of_zeros_with_a_first_weight_below_the_normal_range(T):
    """aa = bb = pp = 0 and u + k around -100: the first denominator is exp(u + k), a number below the smallest
    normal one, and the quotient by it is still v to the few bits that numerator and denominator share."""
    ck = synth_checkpoint(2, 128, vocab=V, seed=31)
    for i in range(2):
        ck[f"blocks.{i}.att.time_first"].fill_(-88.5)
    compare(ck, lambda m, B: torch.zeros_like(m.empty_batch_state(B)), 2, T)


@pytest.mark.parametrize("T", [2, 5, 20, 300, 700])
def test_channels_that_forget_at_once(T):
    """time_decay = 100 overflows to w = -exp(100) = -inf: the state after a step is that step alone."""
    ck = synth_checkpoint(2, 128, vocab=V, seed=31)
    for i in range(2):
        ck[f"blocks.{i}.att.time_decay"][::7] = 100.0
    compare(ck, lambda m, B: m.empty_batch_state(B), 2, T)
