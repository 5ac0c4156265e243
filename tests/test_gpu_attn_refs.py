"""The attention kernel's row references: rows whose scores leave the range that the first tile's reference allows, in either key
half, in both at once, in some rows of a warp only, and by more than the 16-bit or the 32-bit range in one step."""
import pytest
import torch

pytestmark = pytest.mark.gpu

S, SEG = 896, 256


def _levels(pattern, jump):
    """Score (log2 units) of each 64-key half tile."""
    n = S // 64
    j = torch.arange(n)
    tile, half = j // 2, j % 2
    if pattern == "each":
        return jump * j
    if pattern == "first":
        return torch.where(half == 0, jump * tile, torch.zeros_like(j))
    if pattern == "second":
        return torch.where(half == 1, jump * tile, torch.zeros_like(j))
    if pattern == "both":
        return jump * (tile + 2 * half * (tile % 2))
    if pattern == "falling":
        return -jump * j
    if pattern == "late":
        return torch.where(j == n - 3, 6 * jump + 0 * j, torch.zeros_like(j))
    return jump * torch.randint(-2, 4, (n,), generator=torch.Generator().manual_seed(3))


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("dtype,jump", [(torch.bfloat16, 60), (torch.bfloat16, 7), (torch.float16, 20), (torch.float16, 7)])
@pytest.mark.parametrize("pattern", ["each", "first", "second", "both", "falling", "late", "random"])
@pytest.mark.parametrize("rows", ["all", "some"])
def test_rows_that_leave_their_reference(pattern, dtype, jump, head_dim, rows):
    from pbs_attn_b200.prefill import Plan
    g = torch.Generator().manual_seed(1)
    D = head_dim
    u = torch.zeros(D)
    u[: D // 2] = 1.0                                      # the levels live here, the noise of the scores in the other half
    q = torch.randn(1, 1, S, D, generator=g)
    q[..., : D // 2] = 1.0
    if rows == "some":                                     # these see the levels with the other sign, or not at all
        sign = torch.tensor([1.0, -1.0, 0.0])[torch.randint(0, 3, (S,), generator=g)]
        q[..., : D // 2] *= sign[:, None]
    k = torch.randn(1, 1, S, D, generator=g)
    # one key's level: sum of D / 2 equal products, divided by sqrt(D), in log2 units
    unit = D ** 0.5 / 1.4426950408889634 / (D // 2)
    k[..., : D // 2] = (_levels(pattern, jump).float() * unit).repeat_interleave(64)[:, None]
    v = torch.randn(1, 1, S, D, generator=g)
    q, k, v = (t.to(dtype).cuda() for t in (q, k, v))
    plan = Plan(1, 1, 1, S, D, 128, SEG, dtype, q.device)
    plan.segment_permute(k, v, identity=True)
    plan.block_mask.fill_(1)
    plan.build_tile_lists()
    out = torch.full_like(q, float("nan"))
    plan.status.zero_()
    plan.attn_fwd(q, out, attn_impl="tcgen05")
    torch.cuda.synchronize()
    assert not plan.status.any(), plan.status.tolist()
    # blocks of later segments are on in this mask too: every key of the item's lists up to the query counts
    s = q[0, 0].double() @ k[0, 0].double().T / D ** 0.5
    s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    w = torch.softmax(s, -1)
    want, scale = w @ v[0, 0].double(), w @ v[0, 0].double().abs()
    d = (out[0, 0].double() - want).abs()
    # P and the result are rounded to the 16-bit type (8 or 11 significant bits: half a unit is 2^-8 or 2^-11 relative, each; fp16 weights below 2^-14 of their row's reference,
    # which is at most 2^15 below its maximum, to multiples of 2^-25: with 896 keys 2^-15 of the row at most).  A score is exact
    # but for its fp32 sum and the fp32 product and difference of the exponent: magnitudes below 2^11 (in log2 units), a
    # few of their units of 2^-13, so 2^-11 relative in the weights; 2^-10 for both the weight and the sum it is divided by
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    bound = (eps + 2.0 ** -10 + 2.0 ** -14) * scale + eps * want.abs()
    assert (d <= bound).all(), float((d / bound).max())
