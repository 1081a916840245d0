"""The streaming row preparation where its shape changes: one and two input groups per thread (a ragged second
one at 4224 inputs) with the layer norm, two, three and five for plain rows (up to 4096 inputs, up to 6144, beyond
16384; rows_prep_kernel between), CTAs that begin inside a stream."""
import pytest
import torch

from rwkvstic_b200.model import B200RWKV
from rwkvstic_b200.synth import synth_tokens

DEV = "cuda:0"
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("embed", [128, 640, 2560, 3200, 4224, 5120])
def test_rows_path_agrees_with_the_one_row_path_at_every_width(embed):
    model = B200RWKV.synthetic(2, embed, vocab=515, seed=3, device=DEV)
    B, T = 3, 19
    toks = synth_tokens(B * T, seed=embed, vocab=515).reshape(B, T)
    start = model.empty_batch_state(B)
    start[:, :, :2] = torch.randn(start[:, :, :2].shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
    st_rows, st_one = start.clone(), start.clone()
    lg_rows, _ = model.forward_batch(toks, st_rows, rows=True)
    lg_one, _ = model.forward_batch(toks, st_one, rows=False)
    # fp32 statistics summed in another order (a few 2^-24 per layer norm), 24-bit inputs in both
    assert float((lg_rows - lg_one).abs().max()) < 2e-4 * max(1.0, float(lg_one.abs().max()))
    assert torch.allclose(st_rows[:, :, :4], st_one[:, :, :4], rtol=1e-3, atol=2e-4)
    # 450 rows: every CTA takes several, most begin in the middle of a stream; the same bits as one stream alone
    toks = synth_tokens(3 * 150, seed=embed + 1, vocab=515).reshape(3, 150)
    st_all = start.clone()
    lg_all = model.forward_rows(toks, st_all)
    st = start[1:2].clone()
    lg = model.forward_rows(toks[1:2], st)
    assert torch.equal(lg[0], lg_all[1]) and torch.equal(st[0], st_all[1])
    model.check_status()
