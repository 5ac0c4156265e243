"""The register-tiled fp32 attention kernel ("auto") against the generic kernel ("simt") on the same selection."""
import pytest
import torch

from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


# tails of the 32-row query tile and the 64-key step, both head sizes (two buffers / one), both block sizes, one token,
# the dense fallback, rows that keep nothing ("mean" without the own block) and a strided query tensor; 1 to 8 CTAs share a
# query tile (1 from 4500 tokens with 8 heads of 64 on, and at one step), some of them without a step
@pytest.mark.parametrize("tokens,head_dim,block,segment,kind", [
    (1, 64, 64, 64, "pbs"), (33, 64, 64, 128, "pbs"), (250, 128, 128, 256, "pbs"), (640, 64, 64, 128, "pbs"),
    (1500, 64, 128, 256, "strided"), (1023, 128, 64, 64, "pbs"), (2047, 128, 128, 512, "strided"),
    (1500, 64, 64, 64, "mean"), (777, 128, 128, 128, "mean"), (65, 64, 64, 64, "pbs"), (129, 128, 128, 128, "pbs"),
    (4500, 64, 64, 128, "pbs")])
def test_fp32_kernel_equals_generic_kernel(tokens, head_dim, block, segment, kind):
    from pbs_attn_b200.prefill import MeanPooling_prefill, permuted_block_sparse_attn_fwd
    w = Workload("fp32", 2, 4, 2, head_dim, tokens, "fp32", block, segment, 0.7, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=tokens, device="cuda")
    if kind == "strided":
        q, k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v))
    got = []
    for impl in ("auto", "simt"):
        if kind == "mean":
            # 2 is never reached: the rows of heads 0 and 2 keep nothing and come out zero
            thr = torch.tensor([2.0, 0.3, 2.0, 0.6], device="cuda")
            got.append(MeanPooling_prefill(q, k, v, block, segment, thr, force_select_first_block=False,
                                           force_select_current_block=False, attn_impl=impl))
        else:
            got.append(permuted_block_sparse_attn_fwd(q, k, v, block, segment, 0.7, True, attn_impl=impl))
    a, b = (t.double() for t in got)
    if kind == "mean":
        assert not a[:, ::2].any() and not b[:, ::2].any()
    # both sum up to 2047 products of unit size in fp32 (2^-24 relative each, in different orders) and take exp2 of the sums
    assert (a - b).norm() <= 4e-6 * b.norm()
    assert (a - b).abs().max() <= 2e-5


@pytest.mark.parametrize("tokens,head_dim", [(130, 128), (700, 64), (700, 128)])
def test_any_order_of_the_keys(tokens, head_dim):
    """The stage call with an order that crosses segments and all blocks on: plain causal attention."""
    from pbs_attn_b200.prefill import Plan
    w = Workload("order", 1, 4, 2, head_dim, tokens, "fp32", 64, 128, 0.7, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=tokens, device="cuda")
    plan = Plan(1, 4, 2, tokens, head_dim, 64, 128, q.dtype, q.device)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    order = torch.stack([torch.randperm(tokens, generator=g, device="cuda") for _ in range(4)])[None]
    k, v = (t.repeat_interleave(2, dim=1) for t in (k, v))
    plan.key_indices.copy_(order)
    plan.block_mask.fill_(1)
    for dst, src in ((plan.perm_k, k), (plan.perm_v, v)):
        dst.copy_(src.gather(2, order[..., None].expand_as(src)))
    out = torch.empty_like(q)
    plan.attn_fwd(q, out)
    want = torch.nn.functional.scaled_dot_product_attention(q.double(), k.double(), v.double(), is_causal=True)
    # sums of up to 700 products of unit size in fp32 (2^-24 relative each), exp2 of the sums
    assert (out.double() - want).norm() <= 4e-6 * want.norm()
