"""Host-tensor calls of one shape share their staging buffers, whichever stream and thread they are made on."""
import threading

import pytest
import torch

from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


def _inputs(n):
    w = Workload("host", 1, 8, 2, 128, 2048, "bf16", 128, 256, 0.7, 5e5, sinks=4)
    return [[t.pin_memory() for t in make_qkv(w, seed=60 + i)] for i in range(n)]


def _call(x, out=None):
    from pbs_attn_b200.prefill import permuted_block_sparse_attn_fwd_host
    return permuted_block_sparse_attn_fwd_host(*x, 128, 256, 0.7, out=out)


@pytest.mark.parametrize("threads", [False, True])
def test_host_calls_on_several_streams(threads):
    xs = _inputs(3)
    want = []
    for x in xs:
        want.append(_call(x))
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = [[torch.empty_like(w).pin_memory() for _ in range(6)] for w in want]

    def work(i, rounds):
        with torch.cuda.stream(streams[i]):
            for n in rounds:
                _call(xs[i], got[i][n])

    if threads:
        ts = [threading.Thread(target=work, args=(i, range(6))) for i in range(len(xs))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for n in range(6):
            for i in range(len(xs)):
                work(i, [n])
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for gs, w in zip(got, want) for g in gs)


def test_a_call_that_fails_half_way(monkeypatch):
    from pbs_attn_b200 import prefill
    a, b = _inputs(2)
    want = _call(b)
    torch.cuda.synchronize()
    run, calls = prefill.Plan.run, []

    def second_fails(self, *args):
        calls.append(1)
        if len(calls) == 2:
            raise RuntimeError("second chunk")
        return run(self, *args)

    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    monkeypatch.setattr(prefill.Plan, "run", second_fails)
    with torch.cuda.stream(streams[0]), pytest.raises(RuntimeError, match="second chunk"):
        torch.cuda._sleep(50_000_000)
        _call(a)
    with torch.cuda.stream(streams[1]):
        got = _call(b)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
