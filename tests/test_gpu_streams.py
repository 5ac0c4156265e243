"""Calls of one shape on several streams and threads share a plan's scratch: they come one after the other, each with its own result."""
import threading

import pytest
import torch

from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


def _inputs(n, tokens=4096, heads=16):
    w = Workload("streams", 1, heads, 4, 128, tokens, "bf16", 128, 256, 0.7, 5e5, sinks=4)
    return [make_qkv(w, seed=40 + i, device="cuda") for i in range(n)]


def _call(x):
    from pbs_attn_b200.prefill import permuted_block_sparse_attn_fwd
    return permuted_block_sparse_attn_fwd(*x, 128, 256, 0.7, True)


def test_two_streams_in_turn():
    from pbs_attn_b200.prefill import release_plans
    release_plans()
    xs = _inputs(2)
    want = [_call(x).clone() for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = []
    for _ in range(10):
        for x, s in zip(xs, streams):
            with torch.cuda.stream(s):
                got.append(_call(x))
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[i % 2]) for i, g in enumerate(got))


def test_a_plan_that_goes_while_another_stream_uses_it():
    from pbs_attn_b200.prefill import release_plans
    release_plans()
    x, = _inputs(1)
    want = _call(x).clone()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(100_000_000)
        got = _call(x)
    release_plans()
    junk = [torch.full((32 << 20,), 0xFF, dtype=torch.uint8, device="cuda") for _ in range(8)]   # would take over the scratch
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    del junk


def test_threads_with_a_stream_each_and_with_one():
    from pbs_attn_b200.prefill import release_plans
    release_plans()
    xs = _inputs(3, tokens=1024)
    want = [_call(x).clone() for x in xs]
    torch.cuda.synchronize()
    one = torch.cuda.Stream()
    for streams in ([torch.cuda.Stream() for _ in xs], [one] * len(xs)):
        bad = []

        def work(i):
            with torch.cuda.stream(streams[i]):
                got = [_call(xs[i]) for _ in range(50)]
                streams[i].synchronize()
                bad.extend(i for g in got if not torch.equal(g, want[i]))

        threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad
