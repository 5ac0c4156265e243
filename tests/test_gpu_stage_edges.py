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
