"""Rows that see their first key in an entry whose first half raises the references of other rows of the same warp."""
import pytest
import torch

pytestmark = pytest.mark.gpu

H, S = 74, 512


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("dtype,jump", [(torch.bfloat16, 40), (torch.bfloat16, 25), (torch.float16, 20)])
@pytest.mark.parametrize("halves", [(0,), (1,), (0, 1)])
def test_first_reference_beside_a_raise(halves, dtype, jump, head_dim):
    from pbs_attn_b200.prefill import Plan
    D = head_dim
    g = torch.Generator().manual_seed(2)
    # slots 0-127 hold positions 144-271: of the query rows 128-159, a warp, the first half sees no key there, the second half does
    idx = torch.cat([torch.arange(144, 272), torch.arange(0, 144), torch.arange(272, S)])
    q, k, v = (torch.randn(1, H, S, D, generator=g) for _ in range(3))
    q[..., : D // 2] = 1.0
    k[..., : D // 2] = 0.0
    for h in halves:                                       # and then keys that are `jump` (log2 units) above those
        k[:, :, 64 * h : 64 * h + 64, : D // 2] = jump * D ** 0.5 / 1.4426950408889634 / (D // 2)
    q, k, v = (t.to(dtype).cuda() for t in (q, k, v))
    plan = Plan(1, H, H, S, D, 128, S, dtype, q.device)
    plan.key_indices.copy_(idx.int())
    plan.perm_k.copy_(k[:, :, idx])
    plan.perm_v.copy_(v[:, :, idx])
    plan.block_mask.fill_(1)
    plan.build_tile_lists()
    out = torch.empty_like(q)
    for n in range(30):
        got = out if n == 0 else torch.empty_like(q)
        plan.attn_fwd(q, got, attn_impl="tcgen05")
        assert torch.equal(got, out), n                    # whichever warp is first
    plan.check_status()
    s = (q.double() @ k.double().transpose(-1, -2) / D ** 0.5).masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    w = torch.softmax(s, -1)
    want, scale = w @ v.double(), w @ v.double().abs()
    # P and the result in 8 or 11 significant bits; scores below 2^7 log2 units carry a few fp32 units of 2^-17; fp16 weights below 2^-14 of the
    # reference, at most 2^15 below the maximum, are multiples of 2^-24: 2^-25 each, 512 of them 2^-16 of a row
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    bound = (eps + 2.0 ** -13 + 2.0 ** -14) * scale + 2.0 ** -16 + eps * want.abs()
    d = (out.double() - want).abs()
    assert (d <= bound).all(), float((d / bound).max())
