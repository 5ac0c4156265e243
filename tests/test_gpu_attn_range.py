"""The attention kernel at the ends of the range of its operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu

S, D, SEG = 896, 128, 256


def _attend(q, k, v):
    """All blocks on, keys in their order, through the stage calls; q, k, v (S, D)."""
    from pbs_attn_b200.prefill import Plan
    q, k, v = (t[None, None].cuda() for t in (q, k, v))
    plan = Plan(1, 1, 1, S, D, 128, SEG, q.dtype, q.device)
    plan.segment_permute(k, v, identity=True)
    plan.block_mask.fill_(1)
    plan.build_tile_lists()
    out = torch.full_like(q, float("nan"))
    plan.attn_fwd(q, out, attn_impl="tcgen05")
    plan.check_status()
    return out[0, 0].double().cpu()


def _exact(q, k, v):
    s = (q.double() @ k.double().T / D ** 0.5).masked_fill(torch.ones(S, S, dtype=torch.bool).triu(1), float("-inf"))
    w = torch.softmax(s, -1)
    return w @ v.double(), w @ v.double().abs()


@pytest.mark.parametrize("rise", [0, 4, 7, 40, 58])
@pytest.mark.parametrize("exponent", [-118, 100, 114])
def test_large_and_small_values_under_rising_scores(rise, exponent):
    """Scores that rise by `rise` log2 units with every 64 keys: P relative to a row's reference times V must not leave fp32."""
    g = torch.Generator().manual_seed(5)
    q, k = torch.randn(S, D, generator=g), torch.randn(S, D, generator=g)
    unit = D ** 0.5 / 1.4426950408889634 / (D // 2)
    q[:, : D // 2] = 1.0
    k[:, : D // 2] = ((torch.arange(S) // 64).float() * rise * unit)[:, None]
    v = torch.rand(S, D, generator=g) + 0.5
    v *= 2.0 ** exponent * torch.where(torch.rand(S, D, generator=g) < 0.5, -1.0, 1.0)
    q, k, v = (t.bfloat16() for t in (q, k, v))
    got = _attend(q, k, v)
    want, scale = _exact(q, k, v)
    # rounding of P and of the result to 8 significant bits; scores in log2 units below 2^10 carry a few fp32 units of 2^-14: see the
    # derivation for the same scores in test_gpu_attn_refs.py
    bound = (2.0 ** -8 + 2.0 ** -10 + 2.0 ** -14) * scale + 2.0 ** -8 * want.abs()
    assert torch.isfinite(got).all()
    assert ((got - want).abs() <= bound).all(), float(((got - want).abs() / bound).max())


@pytest.mark.parametrize("first", [1e4, 1e7, 1e10])
@pytest.mark.parametrize("level", [-3.0, 0.0, 3.0])
def test_first_keys_far_below_the_others(first, level):
    """The first tile's scores lie `first` (log2 units) below zero, all others near 392 * level / 3: the reference has to reach these."""
    g = torch.Generator().manual_seed(6)
    q, k, v = (torch.randn(S, D, generator=g) for _ in range(3))
    q[:, 0] = 2.0 ** 10
    k[:, 0] = level
    k[:128, 0] = -first / 2.0 ** 10 * D ** 0.5 / 1.4426950408889634
    q, k, v = (t.bfloat16() for t in (q, k, v))
    got = _attend(q, k, v)[128:]                           # (the rows before see nothing else)
    want, scale = (t[128:] for t in _exact(q, k, v))
    # as above: scores of magnitudes below 2^10
    bound = (2.0 ** -8 + 2.0 ** -10 + 2.0 ** -14) * scale + 2.0 ** -8 * want.abs()
    assert ((got - want).abs() <= bound).all(), float(((got - want).abs() / bound).max())
