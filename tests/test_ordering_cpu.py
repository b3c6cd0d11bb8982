"""Memory order of the count that starts the GATED round, read from the kernel's source: the hardware serves the
relaxed form in order too, so no result shows a lost acquire."""
import os
import re

import moe_testlib as tl

SRC = os.path.join(tl.ROOT, "flash_distributed_moe_b200", "csrc", "moe_kernel.cu")


def body_of(name):
    src = re.sub(r"//[^\n]*", "", open(SRC).read())
    start = src.index("{", re.search(r"__forceinline__ \w+ " + name + r"\(", src).end())
    depth = 0
    for i in range(start, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[start:i + 1]


def test_the_last_gated_count_acquires_the_others():
    # one rank: whoever completes the count runs the GATED round, whose threads read the row counts of all workers
    body = body_of("count_gated")
    assert re.search(r"fence_acqrel<\w+>\(\);\s*done = atom_add_acquire\(&p\.peers\[p\.rank\]\.ctl->gated_tokens", body)
    assert "atom.acquire.gpu" in body_of("atom_add_acquire")


def test_the_last_rank_acquires_the_others():
    # several ranks: the same for the count of ranks, before the round is started on the spot
    assert re.search(r"if \(sc && lane == p\.rank\) \{\s*fence_acqrel<S>\(\);\s*sc->run_round2 = 1u;", body_of("gating_finished"))
