"""GPU parity at the edges of the FFN tiles and of the gating rule.  FFN tiles: every token selects the same experts, so that each of them
holds exactly as many (different) rows as there are tokens, and all others none."""
import pytest

import moe_testlib as tl
from moe_testlib import synth
from test_gpu_b_stages import check_layer

pytestmark = pytest.mark.gpu


def same_experts(tokens):
    s = synth.TINY
    gate, w13, w2 = synth.make_weights(s, seed=7, std=0.05)
    x = synth.make_tokens(s, tokens, seed=7)
    x[:, -1] = 1.0
    gate[:, -1] = 0.0
    gate[[3, 11, 18, 30], -1] = tl.torch.tensor([40.0, 36.0, 32.0, 28.0], dtype=gate.dtype)
    return s, x, gate, w13, w2


# one m-tile and two; a wide task's second half with one row, part of a box of rows, and full; a wide task
# of one m-tile behind a full one
@pytest.mark.parametrize("rows", [128, 129, 191, 192, 193, 200, 255, 256, 257, 320, 384, 385])
def test_rows_per_expert_at_the_edges_of_wide_tiles(rows, monkeypatch):
    monkeypatch.setenv("FLASHMOE_WIDE_ROWS", "128")
    s, x, gate, w13, w2 = same_experts(rows)
    check_layer(s, x, gate, w13, w2, max_tokens=rows)


# the edges of the 16-row boxes that tiles of up to 64 rows are loaded in
@pytest.mark.parametrize("rows", [1, 15, 16, 17, 33, 48, 64, 65, 127])
def test_rows_per_expert_at_the_edges_of_row_boxes(rows):
    s, x, gate, w13, w2 = same_experts(rows)
    check_layer(s, x, gate, w13, w2, max_tokens=128)


# on 148 SMs: one token per gating task, two (the last task with one or two), GATE tiles again; and one, two,
# four, eight tokens per COMBINE task
@pytest.mark.parametrize("tokens", [1, 2, 147, 148, 149, 150, 295, 296, 297, 592, 593])
def test_token_counts_at_the_edges_of_the_gating_rule(tokens):
    s = synth.TINY
    gate, w13, w2 = synth.make_weights(s, seed=8, std=0.05)
    check_layer(s, synth.make_tokens(s, tokens, seed=8), gate, w13, w2, max_tokens=max(tokens, 300))


# wide and narrow tiles in one launch, in turn
def test_experts_on_both_sides_of_the_wide_line(monkeypatch):
    monkeypatch.setenv("FLASHMOE_WIDE_ROWS", "128")
    s = synth.TINY
    gate, w13, w2 = synth.make_weights(s, seed=9, std=0.05)
    check_layer(s, synth.make_tokens(s, 1040, seed=9), gate, w13, w2, max_tokens=1040)
