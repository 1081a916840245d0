"""Weights and parameters written by the kernel in front of a call on the same stream are the ones the call uses."""
import ctypes as C

import pytest
import torch

from rwkvstic_b200 import _lib
from rwkvstic_b200.dense_model import B200DenseRWKV
from rwkvstic_b200.model import B200RWKV
from rwkvstic_b200.synth import synth_tokens

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
D = 512


def u8_call(model, tokens, out):
    L = _lib.lib()
    B, T = tokens.shape
    ws = torch.zeros(int(L.b200rwkv_rows_workspace_bytes(C.byref(model._cmodel), B, T)), dtype=torch.uint8, device=DEV)
    state = model.empty_batch_state(B)
    return ws, state, lambda: _lib.check(L.b200rwkv_forward_rows(
        C.byref(model._cmodel), tokens.data_ptr(), B, T, state.data_ptr(), state.stride(0), out.data_ptr(), ws.data_ptr(), ws.numel(),
        torch.cuda.current_stream().cuda_stream))


def dense_call(model, tokens, out):
    L = _lib.lib()
    B, T = tokens.shape
    ws = torch.zeros(int(L.b200rwkv_dense_rows_workspace_bytes(C.byref(model._cmodel), B, T)), dtype=torch.uint8, device=DEV)
    state = model.empty_batch_state(B)
    return ws, state, lambda: _lib.check(L.b200rwkv_dense_forward_rows(
        C.byref(model._cmodel), tokens.data_ptr(), B, T, state.data_ptr(), state.stride(0), out.data_ptr(), ws.data_ptr(), ws.numel(),
        torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("kind", ["u8", "bf16"])
@pytest.mark.parametrize("T", [1, 64])
def test_a_parameter_that_the_call_before_wrote_is_the_one_used(kind, T):
    """The logits of one model are the ln1 weights of another that runs right behind it.  The kernels of a call start
    before their predecessors end and read their parameters then; those of the second call must be the first call's
    result all the same."""
    make = (lambda s: B200RWKV.synthetic(2, D, vocab=D, seed=s, device=DEV, use_graph=False)) if kind == "u8" else \
        (lambda s: B200DenseRWKV.synthetic(2, D, vocab=D, seed=s, dtype=torch.bfloat16, device=DEV, use_graph=False))
    call = u8_call if kind == "u8" else dense_call
    first, second = make(3), make(4)
    tokens = synth_tokens(T, seed=1, vocab=D).reshape(1, T).to(DEV)
    weight = torch.ones(1, D, device=DEV)
    second._clayers[0].ln1_w = weight.data_ptr()
    for _ in range(8):
        a, b = torch.empty(1, D, device=DEV), torch.empty(1, D, device=DEV)
        keep1, _, produce = call(first, tokens, weight)
        keep2, _, use = call(second, tokens, a)
        keep3, _, again = call(second, tokens, b)
        weight.zero_()
        torch.cuda.synchronize()
        produce()
        use()
        torch.cuda.synchronize()
        again()
        torch.cuda.synchronize()
        assert float(weight.abs().max()) > 0 and torch.equal(a, b)
