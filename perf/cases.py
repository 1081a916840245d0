"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is one call of a public entry point on a seeded random-init RWKV-4 model at full depth and with the full
vocabulary, of one of the shapes in ``rwkvstic_b200.synth.SHAPES`` or, for drawn cases, of any size between them:

* ``decode``: every stream takes one token (``B200RWKV.forward`` / ``forward_batch`` for uint8 weights,
  ``B200DenseRWKV.forward`` / ``forward_rows`` for bf16, fp16 and fp32 ones);
* ``prompt``: every stream takes a sequence of tokens (the same entry points in sequence mode);
* ``sample``: one token per row of logits by typical sampling on the device (``ops.sample_typical``).

The weights stand for a loaded checkpoint: they are made once per shape and type and kept by the process, as a
serving program keeps them.  Tokens, the streams' states and logits come from the seed.
"""
from __future__ import annotations

import math
from functools import lru_cache

import torch

from rwkvstic_b200 import ops
from rwkvstic_b200.dense_model import B200DenseRWKV
from rwkvstic_b200.model import B200RWKV
from rwkvstic_b200.synth import SHAPES, VOCAB

DEVICE = "cuda:0"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ITEM = {"u8": 1, "bf16": 2, "fp16": 2, "fp32": 4}


def _net(name, op, shape, weights, streams, tokens):
    layers, embed = SHAPES[shape]
    return {"name": name, "op": op, "layers": layers, "embed": embed, "weights": weights, "streams": streams, "tokens": tokens}


def listed():
    return [
        # A chat or completion loop on the smallest family member: one token at a time, where latency and launches count.
        _net("u8_169m_decode_1", "decode", "169m", "u8", 1, 1),
        # The short prompt in front of such a loop.
        _net("u8_169m_prompt_32", "prompt", "169m", "u8", 1, 32),
        # One user's token loop on a mid-sized and on the headline model: every weight byte is read once per token.
        _net("u8_1b5_decode_1", "decode", "1b5", "u8", 1, 1),
        _net("u8_7b_decode_1", "decode", "7b", "u8", 1, 1),
        # A server's step over many sessions: 256 streams of the headline model, 64 of the largest one.
        _net("u8_7b_decode_256", "decode", "7b", "u8", 256, 1),
        _net("u8_14b_decode_64", "decode", "14b", "u8", 64, 1),
        # One user's prompt of no particular length.
        _net("u8_7b_prompt_333", "prompt", "7b", "u8", 1, 333),
        # A batch of long documents: the largest call.
        _net("u8_3b_prompt_8x1024", "prompt", "3b", "u8", 8, 1024),
        # Unquantised checkpoints: the token loop, a server's step, two long prompts of odd length.
        _net("bf16_7b_decode_1", "decode", "7b", "bf16", 1, 1),
        _net("fp16_1b5_decode_48", "decode", "1b5", "fp16", 48, 1),
        _net("bf16_3b_prompt_2x701", "prompt", "3b", "bf16", 2, 701),
        # The server's sampling of one token for each of 256 sessions.
        {"name": "sample_256", "op": "sample", "rows": 256, "temp": 1.0, "tau": 0.8},
    ]


def _spread(rng, lo, hi):
    """A whole number from lo to hi, uniform in its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _params(layers, embed):
    return 13 * layers * embed * embed


def draw(rng):
    if rng.random() < 0.1:
        return {"op": "sample", "rows": _spread(rng, 1, 256), "temp": round(rng.uniform(0.5, 1.5), 2),
                "tau": round(rng.uniform(0.2, 0.98), 2)}
    weights = rng.choice(["u8"] * 12 + ["bf16"] * 4 + ["fp16"] * 3 + ["fp32"])
    streams = tokens = 1
    op = "decode" if rng.random() < 0.55 else "prompt"
    if op == "decode" and weights != "fp32" and rng.random() < 0.65:
        streams = _spread(rng, 2, 256)
    if rng.random() < 0.6 and weights != "fp32" and not (op == "decode" and streams == 1):
        layers, embed = rng.choice(list(SHAPES.values()))
    else:
        # any member of the family: widths are multiples of 128; fp32 ones only up to the middle of the range
        embed = 128 * _spread(rng, 6, 20 if weights == "fp32" else 40)
        layers = rng.randint(12, 24 if embed < 2048 else 40)
    if op == "prompt":
        rows = _params(*SHAPES["3b"]) * 8192 // _params(layers, embed)       # no more work than the largest listed prompt
        if weights == "fp32":
            tokens = _spread(rng, 2, 12)                                     # fed token by token
        else:
            streams = 1 if rng.random() < 0.6 else rng.randint(2, 8)
            tokens = _spread(rng, 2, min(2048, rows // streams))
    return {"op": op, "layers": layers, "embed": embed, "weights": weights, "streams": streams, "tokens": tokens}


@lru_cache(maxsize=2)
def _model(layers, embed, weights):
    if weights == "u8":
        return B200RWKV.synthetic(layers, embed, device=DEVICE)
    return B200DenseRWKV.synthetic(layers, embed, dtype=DTYPES[weights], device=DEVICE)


def prepare(case, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    if case["op"] == "sample":
        logits = torch.randn(case["rows"], VOCAB, generator=g, device=DEVICE) * 2.0
        u = torch.rand(case["rows"], generator=g, device=DEVICE)
        return {"case": case, "logits": logits, "u": u}
    model = _model(case["layers"], case["embed"], case["weights"])
    B, T, L, D = case["streams"], case["tokens"], model.n_layer, model.n_embd
    tokens = torch.randint(0, VOCAB, (B, T), generator=g, device=DEVICE)
    # Streams in the middle of a text: layer-norm outputs carried over, and weighted sums over past values.
    state = torch.randn(B, L, 5, D, generator=g, device=DEVICE)
    state[:, :, 3] = 1.0 + 9.0 * torch.rand(B, L, D, generator=g, device=DEVICE)
    state[:, :, 2] *= state[:, :, 3]
    if B == 1:
        return {"case": case, "model": model, "tokens": tokens[0], "state": state[0]}
    return {"case": case, "model": model, "tokens": tokens, "state": state}


def run(state):
    case = state["case"]
    if case["op"] == "sample":
        return ops.sample_typical(state["logits"], case["temp"], case["tau"], u=state["u"])
    model = state["model"]
    if case["streams"] == 1:
        logits, new = model.forward(state["tokens"], state["state"])
    elif case["weights"] == "u8":
        logits, new = model.forward_batch(state["tokens"], state["state"])
    else:
        logits, new = model.forward_rows(state["tokens"], state["state"]), state["state"]
    return {"logits": logits, "state": new}


def work(case):
    if case["op"] == "sample":
        n = case["rows"] * VOCAB
        return {"bytes": 4 * n + 12 * case["rows"], "flops": 4 * n}
    layers, embed = case["layers"], case["embed"]
    B, rows = case["streams"], case["streams"] * case["tokens"]
    size = ITEM[case["weights"]]
    matrices = (_params(layers, embed) + VOCAB * embed) * size
    scales = 2 * 4 * (10 * layers * embed + embed) if case["weights"] == "u8" else 0      # one scale and one offset per input
    vectors = 4 * embed * (11 * layers + 4)
    states = 2 * 4 * B * layers * 5 * embed
    ends = 4 * rows * embed + 8 * rows + 4 * B * VOCAB                                   # embedding rows and tokens in, logits out
    return {"bytes": matrices + scales + vectors + states + ends,
            "flops": 2 * (_params(layers, embed) * rows + VOCAB * embed * B)}


def tolerance(case):
    if case["op"] == "sample":
        return {"rel": 1e-6, "differ": 0.01}           # a draw that falls on the edge of two tokens
    # uint8 and fp32: 32-bit sums and vectors through 12 to 40 blocks, the uint8 sums after cancelling their offset.
    # bf16 and fp16: every product is rounded to that type, seven times per block.
    return {"rel": {"u8": 1e-4, "fp32": 2e-5, "bf16": 2e-2, "fp16": 2.5e-3}[case["weights"]]}
