"""The native host side of the common call: same result as the Python one, and back to Python for all that it does not cover."""
import pytest
import torch

from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


def _inputs(dtype="bf16", tokens=700, batch=1, seed=3):
    w = Workload("native", batch, 8, 2, 64, tokens, dtype, 64, 128, 0.8, 5e5, sinks=4)
    return make_qkv(w, seed=seed, device="cuda")


@pytest.mark.parametrize("dtype,tokens,batch", [("bf16", 700, 1), ("fp16", 64, 2), ("fp32", 300, 1), ("bf16", 128, 1)])
@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("mean", [False, True])
def test_same_bits_as_the_python_call(dtype, tokens, batch, strided, mean):
    from pbs_attn_b200 import _cabi
    from pbs_attn_b200.prefill import MeanPooling_prefill, _PLANS, _common_call, permuted_block_sparse_attn_fwd, release_plans
    release_plans()
    q, k, v = _inputs(dtype, tokens, batch)
    if strided:
        q, k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v))
    call = (lambda *a: MeanPooling_prefill(*a, 64, 128, 0.8)) if mean else (lambda *a: permuted_block_sparse_attn_fwd(*a, 64, 128, 0.8, True))
    first = call(q, k, v)                                  # makes the plan: Python
    assert len(_PLANS) == 1
    native = _common_call(q, k, v, 64, 64 if mean else 128, 0.8, True, 2 if mean else 0)
    assert native is not None and native.stride() == first.stride()
    again = call(q, k, v)
    assert torch.equal(native, first) and torch.equal(again, first)
    plan = next(iter(_PLANS.values()))
    assert plan._kv_left_out == (dtype != "fp32" and (mean or tokens <= 128))
    for _ in range(40):                                    # more calls than status slots
        again = call(q, k, v)
    plan.check_status()
    assert torch.equal(again, first)


def test_left_to_python():
    from pbs_attn_b200.prefill import _common_call, permuted_block_sparse_attn_fwd, release_plans
    release_plans()
    q, k, v = _inputs()
    assert _common_call(q, k, v, 64, 128, 0.8, True) is None                      # no plan yet
    want = permuted_block_sparse_attn_fwd(q, k, v, 64, 128, 0.8, True)
    assert torch.equal(_common_call(q, k, v, 64, 128, 0.8, True), want)
    wide = torch.zeros(*q.shape[:3], 65, dtype=q.dtype, device="cuda")[..., :64]   # rows that are not 16-byte aligned
    wide.copy_(q)
    assert _common_call(wide, k, v, 64, 128, 0.8, True) is None
    assert torch.equal(permuted_block_sparse_attn_fwd(wide, k, v, 64, 128, 0.8, True), want)
    assert _common_call(q, k, v, 64, 128, 1, True) is None                        # the int 1 selects everything
    assert _common_call(q, k, v, 64, 128, torch.full((8,), 0.8), True) is None
    assert _common_call(q, k, v.half(), 64, 128, 0.8, True) is None
    assert _common_call(q.cpu(), k.cpu(), v.cpu(), 64, 128, 0.8, True) is None
    assert _common_call(q, k[:, :, :-1], v[:, :, :-1], 64, 128, 0.8, True) is None
    assert _common_call(q, k, v, 64, 96, 0.8, True) is None
    with pytest.raises(AssertionError):
        permuted_block_sparse_attn_fwd(q, k, v, 64, 96, 0.8, True)


def test_plans_that_leave_with_calls_in_flight():
    from pbs_attn_b200.prefill import permuted_block_sparse_attn_fwd, release_plans
    cases = [_inputs(tokens=t, seed=t) for t in (200, 330, 450, 700)]
    release_plans()
    want = [permuted_block_sparse_attn_fwd(*c, 64, 128, 0.8, True) for c in cases]
    for _ in range(5):                                     # four shapes, two plans kept: every call evicts one
        got = [[permuted_block_sparse_attn_fwd(*c, 64, 128, 0.8, True) for _ in range(3)][-1] for c in cases]
    release_plans()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_captured_call_replays():
    from pbs_attn_b200.prefill import permuted_block_sparse_attn_fwd, release_plans
    release_plans()
    q, k, v = _inputs()
    want = permuted_block_sparse_attn_fwd(q, k, v, 64, 128, 0.8, True)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = permuted_block_sparse_attn_fwd(q, k, v, 64, 128, 0.8, True)
    out.zero_()
    g.replay()
    assert torch.equal(out, want)
    assert torch.equal(permuted_block_sparse_attn_fwd(q, k, v, 64, 128, 0.8, True), want)   # plain calls go on
    torch.cuda.synchronize()
    del g
