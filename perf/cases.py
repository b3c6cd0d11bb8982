"""The MoE layer's working range, as cases that can be prepared, run and compared.

A case is one layer shape, one way of calling the launcher and one number of tokens.  `listed()` holds
the calls a serving program makes of this layer: single-token and small-batch decode, ragged chunks,
prefill batches up to the largest, skewed routing, one expert-parallel rank's share of a large layer,
the host-buffer entry point and the fp32 interface.  `draw(rng)` gives more of the same ranges.
"""
import random

import torch

from flash_distributed_moe_b200 import MoeKernelLauncher, synth

# name -> (shape, most tokens of a drawn case): the repository's own layer shapes
LAYERS = {
    "30b": (synth.QWEN3_30B_A3B, 16384),
    "235b": (synth.QWEN3_235B_A22B, 4096),
    "235b-e16": (synth.QWEN3_235B_E16, 4096),
}
SERVING_TOKENS = 8192  # a serving engine creates its launcher once, for its largest batch


def _case(layer, tokens, *, io="bf16", routing="random", max_tokens=None, **name):
    return dict(layer=layer, tokens=tokens, max_tokens=max_tokens or tokens, io=io, routing=routing, **name)


def listed():
    return [
        # one sequence being decoded: eight experts, everything is latency
        _case("30b", 1, max_tokens=SERVING_TOKENS, name="decode_1"),
        # a small decode batch: most experts hold one or two rows
        _case("30b", 16, max_tokens=SERVING_TOKENS, name="decode_16"),
        # a full decode batch (the first benchmark configuration's size): all experts, few rows each
        _case("30b", 128, max_tokens=SERVING_TOKENS, name="decode_128"),
        # a decode batch of the large layer: 4.8 GB of expert weights for 64 tokens
        _case("235b", 64, max_tokens=SERVING_TOKENS, name="decode_64_235b"),
        # the fp32 interface at the size it was made for: fp32 tokens in, fp32 result out
        _case("30b", 48, io="fp32", max_tokens=64, name="fp32_48"),
        # a ragged chunk of a chunked prefill
        _case("30b", 333, max_tokens=SERVING_TOKENS, name="chunk_333"),
        # the benchmark's batch
        _case("30b", 4096, name="prefill_4096"),
        # the same batch when expert popularity follows Zipf(1.2): the hottest experts take every token
        _case("30b", 4096, routing="zipf", name="prefill_4096_zipf"),
        # a long prefill
        _case("30b", 16384, name="prefill_16384"),
        # an ordinary prefill batch of the large layer
        _case("235b", 2048, name="prefill_2048_235b"),
        # the experts of one of eight ranks of the large layer, with an odd number of tokens
        _case("235b-e16", 1531, name="rank_share_1531"),
        # tokens in pinned host memory, result to pinned host memory
        _case("30b", 4096, io="host", name="host_4096"),
    ]


def draw(rng: random.Random):
    io = rng.choice(["bf16"] * 6 + ["host", "fp32"])
    layer = "30b" if io != "bf16" else rng.choice(["30b", "30b", "235b", "235b-e16"])
    most = LAYERS[layer][1] if io == "bf16" else 4096
    tokens = min(most, max(1, round(most ** rng.random())))
    routing = "zipf" if tokens >= 256 and rng.random() < 0.25 else "random"
    max_tokens = max(tokens, rng.choice([tokens, 512, SERVING_TOKENS]))
    return _case(layer, tokens, io=io, routing=routing, max_tokens=max_tokens)


class State:
    """What a program keeps between calls: the launcher with its weights, and the call's buffers."""

    def __init__(self, launcher, weights, tokens, output, host):
        self.launcher, self.weights = launcher, weights
        self.tokens, self.output, self.host = tokens, output, host

    def __del__(self):
        try:
            self.launcher.destroy()
        except Exception:  # the interpreter is going down
            pass


def prepare(case, seed):
    s = LAYERS[case["layer"]][0]
    dtype = torch.float32 if case["io"] == "fp32" else torch.bfloat16
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape, std):  # bf16 values in every case, as a checkpoint holds them
        return torch.empty(*shape, dtype=torch.bfloat16, device=dev).normal_(0.0, std, generator=g)

    gate = normal(s.experts, s.hidden, std=0.02)
    w13 = normal(s.experts, 2 * s.inter, s.hidden, std=0.02).to(dtype)
    w2 = normal(s.experts, s.hidden, s.inter, std=0.02).to(dtype)
    x = normal(case["tokens"], s.hidden, std=1.0)
    if case["routing"] == "zipf":
        gate, x, _ = synth.zipf_routing(s, gate.cpu(), x.cpu(), s=1.2, seed=seed % 65536)
        gate, x = gate.to(dev), x.to(dev)
    weights = (gate.to(dtype), w13, w2)
    launcher = MoeKernelLauncher()
    launcher.create(*weights, case["max_tokens"], launcher.getDistributedUniqueId(empty=True), 0, 1, topk=s.topk)
    host = case["io"] == "host"
    x = x.cpu().pin_memory() if host else x.to(dtype)
    out = torch.empty_like(x, pin_memory=host)
    return State(launcher, weights, x, out, host)


def run(state):
    if state.host:
        state.launcher.launch_host(state.tokens, state.output)
    else:
        state.launcher.launch(state.tokens, state.output)
    return state.output


def work(case):
    s = LAYERS[case["layer"]][0]
    T, H, I, E, K = case["tokens"], s.hidden, s.inter, s.experts, s.topk
    # experts that are selected by at least one of T tokens (each selects K of E)
    active = E * (1.0 - (1.0 - K / E) ** T)
    io = 4 if case["io"] == "fp32" else 2
    return {"bytes": active * 3 * H * I * 2 + E * H * 2 + 2 * T * H * io, "flops": T * (2 * H * E + K * 6 * H * I)}


def tolerance(case):
    # The activations, the weighted expert rows and the result are rounded to bf16.  Against the layer in
    # 64 bits that gives rel 2.9e-3 and max 1.2e-2 to 1.6e-2 over all shapes here; about four times that.
    return {"rel": 1e-2, "max": 6e-2}
