"""Calls whose keys keep their order (the dense fallback, MeanPooling) read K and V where the caller has them; compared
with the generic kernel, which goes through the copy."""
import pytest
import torch

from pbs_attn_b200.synth import Workload, make_qkv

pytestmark = pytest.mark.gpu


def _layout(t, kind):
    if kind == "strided":                       # (B, S, H, D) memory
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    if kind == "heads_first":                   # (H, B, S, D) memory
        return t.transpose(0, 1).contiguous().transpose(0, 1)
    if kind == "wide":                          # rows of a wider matrix, as a fused projection leaves them
        b, h, s, d = t.shape
        big = torch.full((b, s, h * d + 64), float("nan"), dtype=t.dtype, device=t.device)
        view = big[:, :, : h * d].view(b, s, h, d).transpose(1, 2)
        view.copy_(t)
        return view
    return t


# one token, edges of the 128-row tile and of the 256-row group, tails of a block, both block and head sizes
@pytest.mark.parametrize("tokens", [1, 2, 127, 128, 129, 187, 256, 300, 512])
@pytest.mark.parametrize("kind", ["plain", "strided", "heads_first", "wide", "broadcast"])
@pytest.mark.parametrize("call,head_dim,block,segment", [("dense", 128, 128, 512), ("dense", 64, 64, 512), ("dense", 64, 128, 512),
                                                          ("mean", 128, 128, 128), ("mean", 64, 64, 64)])
def test_in_place_equals_copied(tokens, kind, call, head_dim, block, segment):
    from pbs_attn_b200.prefill import MeanPooling_prefill, permuted_block_sparse_attn_fwd
    w = Workload("inplace", 2, 4, 2, head_dim, tokens, "bf16", block, segment, 0.7, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=tokens, device="cuda")
    if kind == "broadcast":                     # a zero head stride: the copy is kept
        k, v = k[:, :1].expand(-1, 2, -1, -1), v[:, :1].expand(-1, 2, -1, -1)
    else:
        q, k, v = (_layout(t, kind) for t in (q, k, v))
    got, inters = [], []
    for impl in ("tcgen05", "simt"):
        inter = {}
        if call == "mean":
            got.append(MeanPooling_prefill(q, k, v, block, segment, 0.7, attn_impl=impl, intermediates=inter))
        else:
            got.append(permuted_block_sparse_attn_fwd(q, k, v, block, segment, 0.7, True, attn_impl=impl, intermediates=inter))
        inter["plan"].check_status()
        inters.append((inter["key_indices"].clone(), inter["block_mask"].clone(), inter["plan"].first_block.clone()))
    assert all(torch.equal(a, b) for a, b in zip(*inters))
    d = (got[0].float() - got[1].float()).abs()
    # P and the result are rounded to bf16 in both (2^-9 relative each); |v| stays below 6
    assert torch.isfinite(d).all() and d.max() <= 5e-2 and d.mean() <= 2e-3
