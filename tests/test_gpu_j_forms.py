"""GPU: the other forms that a launch on one GPU can take (GATE and DISPATCH tiles at few tokens, wide FFN tiles at
few rows, publication batches), asked for by environment variables, over what the default forms are tested on."""
import numpy as np
import pytest
import torch

import moe_testlib as tl
import test_gpu_b_stages as stages
import test_gpu_c_api as api
from moe_testlib import cpu_oracle, synth

pytestmark = pytest.mark.gpu

DISPATCH, FFN1 = 9, 1  # task kinds in the event trace


def tasks_run(layer):
    """Kinds of the tasks of the only launch of a layer created with FLASHMOE_PROFILE=1, with their number."""
    ev = np.frombuffer(layer.launcher.debug_read(8, layer.grid * 512 * 16), np.uint32).reshape(layer.grid, 512, 4)
    kinds = np.concatenate([ev[b, 1:1 + ev[b, 0, 0], 0] for b in range(layer.grid)])
    return dict(zip(*[v.tolist() for v in np.unique(kinds, return_counts=True)]))


def weighted_rows(layer, tokens):
    s = layer.shape
    return np.frombuffer(layer.launcher.debug_read(6, tokens * s.topk * s.hidden * 2), np.int16).copy()


def new_layer(s, weights, tokens, monkeypatch, **env):
    for k, v in env.items():
        monkeypatch.setenv(k, str(v))
    return tl.GpuLayer(s, *weights, tokens)


# on 148 SMs, the rule's line is at 296 tokens
@pytest.mark.parametrize("tokens, gate_rows, tiles", [(148, 0, 0), (296, 0, 0), (297, 0, 10), (148, 32, 5), (1, 32, 1),
                                                      (300, 2, 0), (300, 1, 10)])
def test_the_form_of_the_gating_follows_the_rule_and_the_variable(tokens, gate_rows, tiles, monkeypatch):
    s = synth.TINY
    layer = new_layer(s, synth.make_weights(s, seed=20, std=0.05), 300, monkeypatch, FLASHMOE_PROFILE=1,
                      FLASHMOE_GATE_ROWS=gate_rows)
    try:
        if layer.grid != 148:
            pytest.skip("token counts are those of 148 SMs")
        layer.run(synth.make_tokens(s, tokens, seed=20))
        assert tasks_run(layer).get(DISPATCH, 0) == tiles
    finally:
        layer.close()


# tests of small launches, whose tokens GATE tiles of one or two send themselves, with GATE tiles of 32 and
# DISPATCH: stage by stage, all tied, in place, repeated, from host buffers, fp32, replayed from a graph
@pytest.mark.parametrize("test", [
    stages.test_tiny_layer_ragged_tokens, stages.test_qwen3_30b_reference_test_stream_48_tokens_in_place,
    stages.test_all_logits_tied_every_token_takes_the_exact_path, stages.test_qwen3_235b_sizes_ragged_tokens,
    stages.test_qwen3_235b_sizes_golden_24_tokens_in_place, api.test_zero_tokens_and_repeated_launches,
    api.test_host_buffer_entry_point_matches_device_entry_point,
    api.test_host_entry_point_pipelines_back_to_back_calls, api.test_fp32_io_adapter,
    api.test_block_wrapper_in_place, api.test_single_gpu_launch_replays_from_a_cuda_graph,
], ids=lambda t: t.__name__)
def test_few_tokens_through_gate_and_dispatch_tiles(test, monkeypatch):
    monkeypatch.setenv("FLASHMOE_GATE_ROWS", "32")
    test()


def test_one_launcher_in_place_across_the_forms_of_gating():
    s = synth.TINY
    gate, w13, w2 = synth.make_weights(s, seed=21, std=0.05)
    x = synth.make_tokens(s, 600, seed=21)
    ref = cpu_oracle.PortOracle().full_moe(tl.f32(x), tl.f32(gate), tl.f32(w13), tl.f32(w2), s.topk)
    layer = tl.GpuLayer(s, gate, w13, w2, 600)
    try:
        for tokens in (600, 1, 333, 296, 297, 2, 148, 600):
            tl.assert_close_bf16(tl.f32(layer.run(x[:tokens], inplace=True)), ref[:tokens], f"{tokens} tokens")
    finally:
        layer.close()


# wide tiles in launches that the rule gives narrow ones: five m-tiles per expert at hidden 4096, exactly full buffers
@pytest.mark.parametrize("test", [
    stages.test_qwen3_235b_sizes_many_tiles_per_expert,
    stages.test_qwen3_30b_zipf_routing_hottest_expert_takes_every_token,
], ids=lambda t: t.__name__)
def test_wide_tiles_against_the_oracle(test, monkeypatch):
    monkeypatch.setenv("FLASHMOE_WIDE_ROWS", "128")
    test()


# 16 experts of 12 and 16 n-tiles, rows per expert around 128, 192 (the second half's tile is transposed up to
# there), 256 and 765; on 12 workers, so that each runs dozens of wide tasks one behind another, and narrow ones of the experts
# with up to 128 rows in between.  Narrow and wide tiles add the same products in the same order.
@pytest.mark.parametrize("tokens", [256, 384, 512, 1531])
def test_wide_tiles_one_behind_another_have_the_bits_of_narrow_ones(tokens, monkeypatch):
    s = synth.QWEN3_235B_E16
    weights = synth.make_weights(s, seed=22)
    x = synth.make_tokens(s, tokens, seed=22)
    layer = new_layer(s, weights, tokens, monkeypatch, FLASHMOE_WIDE_ROWS=1 << 30)
    try:
        out, y = layer.run(x), weighted_rows(layer, tokens)
        cnt = np.frombuffer(layer.launcher.debug_read(2, s.experts * 4), np.uint32).astype(int)
    finally:
        layer.close()
    layer = new_layer(s, weights, tokens, monkeypatch, FLASHMOE_WIDE_ROWS=128, FLASHMOE_GRID=12, FLASHMOE_PROFILE=1)
    try:
        assert layer.grid == 12
        for i in range(2):
            got = layer.run(x)
            if i == 0:
                assert tasks_run(layer)[FFN1] == 12 * sum(-(-c // 256) for c in cnt)
            assert np.array_equal(weighted_rows(layer, tokens), y)
            assert torch.equal(got.view(torch.int16), out.view(torch.int16))
    finally:
        layer.close()
    assert tokens != 256 or ((cnt <= 128).any() and (cnt > 128).any())


# experts with exactly as many rows as there are tokens and weights that all count: the weighted rows slot by slot
@pytest.mark.parametrize("rows", [129, 192, 193, 256, 257, 385])
def test_weighted_rows_of_wide_tiles_slot_by_slot(rows, monkeypatch):
    s = synth.TINY
    gate, w13, w2 = synth.make_weights(s, seed=23, std=0.05)
    x = synth.make_tokens(s, rows, seed=23)
    x[:, -1] = 1.0
    gate[:, -1] = 0.0
    gate[[3, 11, 18, 30], -1] = torch.tensor([40.0, 39.5, 39.0, 38.5], dtype=gate.dtype)
    port = cpu_oracle.PortOracle()
    _, w, _, _, y = port.full_moe(tl.f32(x), tl.f32(gate), tl.f32(w13), tl.f32(w2), s.topk, stages=True)
    layer = new_layer(s, (gate, w13, w2), rows, monkeypatch, FLASHMOE_WIDE_ROWS=128)
    try:
        layer.run(x)
        got = tl.f32(layer.stages(rows)["y"])
    finally:
        layer.close()
    for k in range(s.topk):
        tl.assert_close_bf16(got[:, k], (y * w[:, :, None])[:, k], f"slot {k}")


# FFN1 tiles published while rows are still arriving: one GPU does without, several ranks do it
@pytest.mark.parametrize("batch_mt", [1, 2])
@pytest.mark.parametrize("wide_rows", [128, 1 << 30])
def test_publication_batches_on_one_gpu(batch_mt, wide_rows, monkeypatch):
    monkeypatch.setenv("FLASHMOE_BATCH_MT", str(batch_mt))
    monkeypatch.setenv("FLASHMOE_WIDE_ROWS", str(wide_rows))
    s = synth.TINY
    gate, w13, w2 = synth.make_weights(s, seed=24, std=0.05)
    for tokens in (200, 3000):
        stages.check_layer(s, synth.make_tokens(s, tokens, seed=24), gate, w13, w2, max_tokens=3000)
