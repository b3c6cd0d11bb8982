"""GPU: a token's result has the same bits in any batch on one GPU, whatever the size of the GATE tile it falls into,
nearly tied or not."""
import numpy as np
import pytest
import torch

import moe_testlib as tl
from moe_testlib import synth
from test_gpu_b_stages import check_layer

pytestmark = pytest.mark.gpu

# many experts over small FFNs: more of them may be nearly tied than one task regates
MANY = synth.LayerShape("many-experts", 2048, 128, 128, 8)


def routing(layer, T):
    K = layer.shape.topk
    return (np.frombuffer(layer.launcher.debug_read(0, T * K * 4), np.int32).reshape(T, K).copy(),
            np.frombuffer(layer.launcher.debug_read(1, T * K * 4), np.uint32).reshape(T, K).copy())


def inputs_with_ties(s, tokens, seed):
    """Beside the near-ties of random logits: two pairs of experts with equal gate rows, so that a token with one of
    a pair among its leading logits is tied, and rows of zeros, all of whose logits are tied.  GATE tiles of two
    tokens see each kind in neither, one, the other and both of their tokens."""
    gate, w13, w2 = synth.make_weights(s, seed=seed, std=0.05 if s is synth.TINY else 0.02)
    x = synth.make_tokens(s, tokens, seed=seed)
    gate[5], gate[s.experts - 1] = gate[4], gate[s.experts - 2]
    for t in (1, 6, 7, 12, 90, 151, 152, 153):
        if t < tokens:
            x[t] = 0.0
    return x, gate, w13, w2


# on 148 SMs: GATE tiles of 32 tokens (600), of one token (up to 148), of two (149 to 296, the last one with
# one token or two), of 32 again
@pytest.mark.parametrize("s", [synth.TINY, MANY, synth.QWEN3_235B_E16], ids=lambda s: s.name)
def test_a_token_gives_the_same_bits_in_any_batch(s):
    x, gate, w13, w2 = inputs_with_ties(s, 600, seed=11)
    layer = tl.GpuLayer(s, gate, w13, w2, 600)
    try:
        out = layer.run(x)
        idx, w = routing(layer, 600)
        for n in (1, 2, 37, layer.grid, layer.grid + 1, 2 * layer.grid - 1, 2 * layer.grid, 2 * layer.grid + 1):
            got = layer.run(x[:n], inplace=True)
            gi, gw = routing(layer, n)
            assert np.array_equal(gi, idx[:n]) and np.array_equal(gw, w[:n]), f"routing of {n} tokens"
            assert torch.equal(got.view(torch.int16), out[:n].view(torch.int16)), f"output of {n} tokens"
    finally:
        layer.close()


@pytest.mark.parametrize("gate_rows", [1, 2, 64, 128])
def test_the_size_of_the_gate_tiles_does_not_change_a_bit(gate_rows, monkeypatch):
    x, gate, w13, w2 = inputs_with_ties(synth.TINY, 145, seed=12)
    layer = tl.GpuLayer(synth.TINY, gate, w13, w2, 145)
    try:
        monkeypatch.setenv("FLASHMOE_GATE_ROWS", "32")
        out, (idx, w) = layer.run(x), routing(layer, 145)
        monkeypatch.setenv("FLASHMOE_GATE_ROWS", str(gate_rows))
        got, (gi, gw) = layer.run(x), routing(layer, 145)
        assert np.array_equal(gi, idx) and np.array_equal(gw, w)
        assert torch.equal(got.view(torch.int16), out.view(torch.int16))
    finally:
        layer.close()


@pytest.mark.parametrize("tokens", [13, 154])
@pytest.mark.parametrize("s", [synth.TINY, MANY], ids=lambda s: s.name)
def test_tied_tokens_of_small_gate_tiles_against_the_oracle(s, tokens):
    check_layer(s, *inputs_with_ties(s, tokens, seed=13), max_tokens=tokens)
