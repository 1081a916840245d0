"""The WKV scan of the prompt path where its chunks and its arithmetic can go wrong, against the one-row path (one
token at a time, the same fp32 recurrence step by step)."""
import pytest
import torch

from oracle.fastquant_oracle import OracleRWKV
from oracle.torch_mode_oracle import OracleTorchMode
from rwkvstic_b200.dense_model import B200DenseRWKV
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


LONG = [513, 700, 1025]      # more than the 32 warps of a CTA take in one turn (16 steps each): two and three turns


@pytest.mark.parametrize("T", LONG + [512, 511])
def test_one_long_stream(T):
    """One stream of 2560 channels is 80 CTAs of 32 warps, two are 160 of 16 (more than one per SM): the carried state
    goes through both groups of 16 warps in the first and through one in the second.  Against the oracle's sequence
    mode, and bit for bit against the same stream beside another one."""
    D, W = 2560, 300
    ck = synth_checkpoint(1, D, vocab=W, seed=77)
    ref = OracleRWKV(ck)
    model = B200RWKV.from_checkpoint(ck, device=DEV, use_graph=False)
    model.rows_per_call = 4096
    tokens = synth_tokens(2 * T, seed=T, vocab=W).reshape(2, T)
    both, alone = model.empty_batch_state(2), model.empty_batch_state(1)
    lg_both = model.forward_rows(tokens, both)
    lg_alone = model.forward_rows(tokens[:1], alone)
    assert torch.equal(lg_alone[0], lg_both[0]) and torch.equal(alone[0], both[0])
    want, state = ref.forward(tokens[0], ref.emptyState.clone())
    assert float((lg_alone[0].cpu().double() - want).abs().max()) < 2e-3
    # the same allowance as test_chunked_wkv_scan_at_1024_tokens_against_the_oracle
    mine, ref4 = model.to_reference_state(alone[0]).cpu()[:, :4], state[:, :4]
    excess = (mine - ref4).abs() - (2e-4 + 2e-3 * ref4.abs() + 2e-5 * ref4.abs().amax(dim=2, keepdim=True))
    assert float(excess.max()) <= 0
    model.check_status()


@pytest.mark.parametrize("T", LONG)
def test_one_long_stream_of_the_16_bit_path(T):
    """The scan that writes 16-bit rows, over two and three turns of 32 warps, against the oracle."""
    D, W = 2560, 300
    ck = synth_checkpoint(1, D, vocab=W, seed=78)
    ref = OracleTorchMode(ck, torch.bfloat16)
    model = B200DenseRWKV.from_checkpoint(ck, dtype=torch.bfloat16, device=DEV, use_graph=False)
    tokens = synth_tokens(T, seed=T, vocab=W)
    state = model.empty_batch_state(1)
    out = model.forward_rows(tokens.reshape(1, T), state)
    want, wstate = ref.forward(tokens, ref.emptyState.clone())
    # one block of products rounded to 8 significant bits: four units of the last place of the largest logit, as the
    # smoke check allows
    assert float((out[0].cpu() - want).abs().max()) <= 4 * 2.0 ** -8 * float(want.abs().max())
    # sums of values that carry the same rounding, over the state's own scale
    for row in (2, 3):
        a, b = state[0, 0, row].cpu(), wstate[0, row]
        scale = torch.exp(state[0, 0, 4].cpu() - wstate[0, 4])          # both are relative to their largest exponent
        assert float((a * scale - b).norm() / b.norm()) <= 2.0 ** -8
    model.check_status()
