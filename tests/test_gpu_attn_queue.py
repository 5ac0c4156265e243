"""The attention kernel's work queue: every (head, query group) is computed exactly once at item counts around
the number of CTAs and of whole waves of pairs, and the draw counter in the status words is zero again afterwards."""
import pytest
import torch

from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


# 256-query groups per head x heads: below one item a CTA, one wave of items, odd group counts, whole waves of
# pairs (148 SMs: 8 x 37 = 296, 74 x 8 = 592 items), whole waves and a rest, and a first head the pairs take in part
@pytest.mark.parametrize("groups,heads", [(1, 3), (3, 5), (4, 37), (5, 29), (8, 37), (7, 43), (74, 8), (9, 70), (23, 40)])
def test_every_item_once_and_counter_back_at_zero(groups, heads):
    from pbs_attn_b200.prefill import Plan
    S = groups * 256 - 40
    w = Workload("queue", 1, heads, 1, 64, S, "bf16", 64, 128, 0.8, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=groups, device="cuda")
    plan = Plan(1, heads, 1, S, 64, 64, 128, q.dtype, q.device)
    first, again, generic = (torch.full_like(q, float("nan")) for _ in range(3))
    plan.run(q, k, v, first, plan.options(0.8, attn_impl="tcgen05"))
    plan.check_status()
    assert not plan.status.any()
    plan.run(q, k, v, again, plan.options(0.8, attn_impl="tcgen05"))
    plan.run(q, k, v, generic, plan.options(0.8, attn_impl="simt"))
    torch.cuda.synchronize()
    plan.check_status()
    assert torch.equal(first, again)
    d = (first.float() - generic.float()).abs()
    # both kernels round P and the result to bf16 (2^-9 relative each); a row attends to 128 keys or more of unit variance
    assert torch.isfinite(d).all() and d.max() <= 2e-2 and d.mean() <= 1e-3
