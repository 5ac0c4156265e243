"""The stages before the attention at the edges of their dispatch: statistics of few and many tiles, 8 and 16 rows per
CTA in the selection, and pooling at block sizes that do not divide 256."""
import pytest
import torch

from oracle import pbs_oracle
from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


def _inputs(dtype, heads, D, tokens, block, segment, seed=0):
    w = Workload("edge", 1, heads, 1, D, tokens, dtype, block, segment, 0.8, 5e5, sinks=4)
    return make_qkv(w, seed=seed, device="cuda")


# 64-key tiles: 1, 31, 32, 33, 128 (last of the one-warp merge), 129, 200
@pytest.mark.parametrize("tiles", [1, 31, 32, 33, 128, 129, 200])
@pytest.mark.parametrize("dtype,D", [("bf16", 128), ("fp16", 128), ("fp16", 64)])
def test_importance_is_the_softmax_of_its_own_logits(tiles, dtype, D):
    from pbs_attn_b200.prefill import Plan
    S = 64 * tiles + 10
    q, k, _ = _inputs(dtype, 2, D, S, 64, 64)
    plan = Plan(1, 2, 1, S, D, 64, 64, q.dtype, q.device)
    imp, logits = plan.key_importance(q, k, want_logits=True)
    want = torch.softmax(logits.double(), dim=-1).mean(dim=-2)
    # fp32 sums of up to 12810 exponentials taken in runs, one exponential and one quotient per term: a few 2^-22
    assert ((imp.double() - want).abs() <= 2e-6 * want).all()


# 8-row CTAs up to 444 of them (148 SMs), 16-row CTAs beyond (nb <= 256), and the larger register counts; pooled rows of
# 8, 16 and 32 16-byte pieces
@pytest.mark.parametrize("heads,nb", [(1, 3), (27, 128), (28, 128), (55, 64), (56, 64), (13, 256), (14, 256), (2, 300), (2, 600), (1, 1030)])
@pytest.mark.parametrize("thr", [0.0, 0.3, 0.9, 1.0, 2.0])
@pytest.mark.parametrize("dtype,D,diagonal", [(torch.bfloat16, 64, False), (torch.bfloat16, 128, False), (torch.float16, 128, True),
                                              (torch.bfloat16, 256, True), (torch.float32, 64, True), (torch.float32, 128, False)])
def test_selection_equals_the_general_kernel(heads, nb, thr, dtype, D, diagonal):
    from pbs_attn_b200 import _cabi
    from pbs_attn_b200.prefill import Plan
    lib = _cabi.load()
    plan = Plan(1, heads, 1, nb * 64 - 7, D, 64, 128, dtype, "cuda")
    g = torch.Generator(device="cuda").manual_seed(nb)
    plan.pooled_q.copy_(torch.randn(plan.pooled_q.shape, generator=g, device="cuda"))
    plan.pooled_k.copy_(torch.randn(plan.pooled_k.shape, generator=g, device="cuda").round())    # ties among the scores
    plan.first_block.zero_()
    got = []
    try:
        for impl in (0, 1):
            lib.pbs_debug_set_select_impl(impl)
            scores = plan.select_blocks(plan.options(thr, diagonal_candidates=diagonal), want_scores=True)
            got.append((plan.block_mask.clone(), scores))
    finally:
        lib.pbs_debug_set_select_impl(0)
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("block", [16, 48, 96, 128, 240, 256])
@pytest.mark.parametrize("dtype,D", [("bf16", 128), ("fp16", 8), ("fp32", 64), ("fp32", 256)])
@pytest.mark.parametrize("mode", ["mean", "max"])
def test_pooled_keys_equal_the_reference_order(block, dtype, D, mode):
    from pbs_attn_b200.prefill import Plan
    S, segment = 3 * 4 * block + block + 5, 4 * block
    q, k, v = _inputs(dtype, 2, D, S, block, segment)
    plan = Plan(1, 2, 1, S, D, block, segment, q.dtype, q.device)
    plan.segment_permute(k, v, mode, identity=True)
    want = pbs_oracle._pool(pbs_oracle._pad_to_block(pbs_oracle.repeat_kv(k.cpu(), 2), block), block, mode)
    assert torch.equal(plan.perm_k.cpu(), pbs_oracle.repeat_kv(k.cpu(), 2)) and torch.equal(plan.perm_v.cpu(), pbs_oracle.repeat_kv(v.cpu(), 2))
    assert torch.equal(plan.pooled_k.cpu(), want)
