"""The attention kernel's work queue: every (head, query group) is computed at item counts around the number of CTAs and of
whole waves of pairs, and the draw counter in the status words is zero again afterwards.  (That no item is in two entries of
the queue is shown on the host, in test_attn_schedule.py.)"""
import pytest
import torch

from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


# 256-query groups per head x heads: below one item a CTA, one wave of items, odd group counts, whole waves of
# pairs (148 SMs: 8 x 37 = 296, 74 x 8 = 592 items), whole waves and a rest, and a first head the pairs take in part
@pytest.mark.parametrize("groups,heads", [(1, 3), (3, 5), (4, 37), (5, 29), (8, 37), (7, 43), (74, 8), (9, 70), (23, 40)])
def test_every_item_and_counter_back_at_zero(groups, heads):
    from pbs_attn_b200.prefill import Plan
    S = groups * 256 - 40
    w = Workload("queue", 1, heads, 1, 64, S, "bf16", 64, 128, 0.8, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=groups, device="cuda")
    plan = Plan(1, heads, 1, S, 64, 64, 128, q.dtype, q.device)
    first, again, generic, scale = (torch.full_like(q, float("nan")) for _ in range(4))
    plan.run(q, k, v, first, plan.options(0.8, attn_impl="tcgen05"))
    plan.check_status()
    assert not plan.status.any()
    plan.run(q, k, v, again, plan.options(0.8, attn_impl="tcgen05"))
    plan.run(q, k, v, generic, plan.options(0.8, attn_impl="simt"))
    plan.run(q, k, v.abs(), scale, plan.options(0.8, attn_impl="simt"))
    torch.cuda.synchronize()
    plan.check_status()
    assert torch.equal(first, again)
    d = (first.float() - generic.float()).abs()
    # both kernels round P and the result to bf16, 2^-8 relative each: with sum P |v| = scale they differ by no more than
    # 2 * 2^-8 (scale + |result|), and scale is itself rounded twice
    assert (d <= 2.0 ** -7 * 1.02 * (scale.float() + generic.float().abs())).all() and d.mean() <= 1e-3


# 512 items, more than three waves of CTAs
def test_stage_call_needs_no_words_of_its_own():
    """pbs_attn_fwd on status words that an earlier call left behind, and twice at once on one set of them."""
    from pbs_attn_b200 import _cabi
    from pbs_attn_b200.prefill import Plan, _ptr, _strides
    S, H = 4096, 32
    w = Workload("words", 1, H, 8, 128, S, "bf16", 128, 256, 0.8, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=5, device="cuda")
    plan = Plan(1, H, 8, S, 128, 128, 256, q.dtype, q.device)
    want = plan.run(q, k, v, torch.empty_like(q), plan.options(0.8, attn_impl="tcgen05"))
    plan.check_status()

    def stage(words, stream):
        out = torch.full_like(q, float("nan"))
        stream.wait_stream(torch.cuda.current_stream())
        _cabi.check(plan.lib.pbs_attn_fwd(_cabi.C.byref(plan.shape), _ptr(q), _strides(q), _ptr(plan.perm_k), _ptr(plan.perm_v),
                                          _ptr(plan.key_indices), _ptr(plan.block_mask), _ptr(plan.tile_list), _ptr(plan.tile_count),
                                          _ptr(out), _strides(out), _cabi.ATTN_IMPL["tcgen05"], _ptr(words), None,
                                          _cabi.C.c_void_p(stream.cuda_stream)), "pbs_attn_fwd")
        return out

    left = torch.tensor([0] + [5] * 7, dtype=torch.int32, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [stage(left, streams[0])]
    torch.cuda.synchronize()
    shared = torch.zeros(8, dtype=torch.int32, device="cuda")
    outs += [stage(shared, s) for s in streams for _ in range(4)]
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
    assert left.tolist() == [0] + [5] * 7 and not shared.any()
