"""Where a plan may be made: under a capture, and on a device that is not the current one."""
import os
import subprocess
import sys

import pytest
import torch

from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


def _inputs(tokens, device="cuda"):
    return make_qkv(Workload("attach", 1, 8, 2, 64, tokens, "bf16", 64, 128, 0.8, 5e5, sinks=4), seed=9, device=device)


@pytest.mark.parametrize("leaving", [False, True])
def test_first_call_of_a_shape_under_capture(leaving):
    from pbs_attn_b200.prefill import permuted_block_sparse_attn_fwd, release_plans
    x, other = _inputs(700), _inputs(300)
    want = permuted_block_sparse_attn_fwd(*x, 64, 128, 0.8, True)
    torch.cuda.synchronize()
    release_plans()
    if leaving:                                            # a plan that goes with a call in flight
        torch.cuda._sleep(200_000_000)
        permuted_block_sparse_attn_fwd(*other, 64, 128, 0.8, True)
        release_plans()
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):                             # (torch.cuda.graph would wait for the call in flight first)
        g.capture_begin()
        out = permuted_block_sparse_attn_fwd(*x, 64, 128, 0.8, True)
        g.capture_end()
    torch.cuda.synchronize()
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    release_plans()
    del g


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two devices")
def test_a_process_on_the_second_device_leaves_the_first_alone():
    code = ("import torch\nfrom pbs_attn_b200.prefill import permuted_block_sparse_attn_fwd as f\n"
            "x = [torch.randn(1, 2, 300, 64, device='cuda:1').bfloat16() for _ in range(3)]\nf(*x, 64, 128, 0.8, True)\n"
            "torch.cuda.synchronize(1)\nassert not torch._C._cuda_hasPrimaryContext(0)")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], cwd=root, check=True, timeout=300)
