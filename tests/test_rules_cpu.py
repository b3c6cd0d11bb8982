"""Host rules that choose how a launch on one GPU is cut (csrc/host_layout.h), over every token count, checked
by a small C++ program against the counters and queue slots the launch has.  No GPU."""
import os
import subprocess

import moe_testlib as tl

CSRC = os.path.join(tl.ROOT, "flash_distributed_moe_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_rules_fit_the_counters_and_queues(tmp_path):
    exe = str(tmp_path / "rules_test.bin")
    src = os.path.join(tl.ROOT, "tests", "cpp", "rules_test.cpp")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, src, f"-I{CUDA}/include", f"-I{CSRC}"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
