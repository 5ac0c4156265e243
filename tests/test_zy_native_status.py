"""Status words of calls that run without Python: a call whose wait ran out is reported, and the words of calls that are still
in flight when their plan goes reach nobody else.  (How a wait is made to run out: test_zy_failure_path.py.)"""
import time

import pytest
import torch

from pbs_attn_b200 import _cabi
from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


def _calls(tokens, seed):
    from pbs_attn_b200.prefill import permuted_block_sparse_attn_fwd
    w = Workload("status", 1, 4, 1, 128, tokens, "bf16", 128, 256, 0.9, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=seed, device="cuda")
    return lambda: permuted_block_sparse_attn_fwd(q, k, v, 128, 256, 0.9, True)


def _failing(call):
    lib = _cabi.load()
    try:
        assert lib.pbs_debug_set_attn_wait(3_000_000, 1) == 0
        call()
    finally:
        assert lib.pbs_debug_set_attn_wait(0, 0) == 0


def test_a_call_without_python_reports_its_wait():
    from pbs_attn_b200.prefill import _PLANS, release_plans
    release_plans()
    call = _calls(2048, 5)
    good = call()
    assert torch.equal(call(), good)                       # (this one ran without Python)
    _failing(call)
    torch.cuda.synchronize()
    with pytest.raises(_cabi.PbsError, match="bounded wait"):
        call()
    with pytest.raises(_cabi.PbsError):
        next(iter(_PLANS.values())).check_status()
    for _ in range(20):
        again = call()
    next(iter(_PLANS.values())).check_status()
    assert torch.equal(again, good)


def test_words_that_land_late_reach_no_other_plan():
    from pbs_attn_b200.prefill import release_plans
    release_plans()
    a, b = _calls(2048, 6), _calls(1024, 7)
    torch.cuda.synchronize()
    s, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(1000)
        a()
        s.synchronize()
        torch.cuda._sleep(200_000_000)                     # a tenth of a second, so that both calls are made before the first ends
        _failing(a)
        torch.cuda._sleep(2_000_000_000)                   # a second
        later = a()
        time.sleep(0.3)                                    # the failing call's words are there, those of the last one are not
        with pytest.raises(_cabi.PbsError, match="bounded wait"):
            a()
    behind = torch.cuda.Event()
    behind.record(s)
    release_plans()
    with torch.cuda.stream(s2):
        b(), b()
        _failing(b)
    s2.synchronize()
    assert not behind.query()                              # the words of a's last call are still to come
    torch.cuda.synchronize()
    with torch.cuda.stream(s2), pytest.raises(_cabi.PbsError, match="bounded wait"):
        b()
    del later
    release_plans()
