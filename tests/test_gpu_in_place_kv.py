"""Calls whose keys keep their order (the dense fallback, MeanPooling) read K and V where the caller has them; compared
with the same call through the copies, and with the generic kernel."""
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


def _same_but_for_rounding(a, b, scale):
    """P and the result are rounded to bf16 in both, 2^-8 relative each: with sum P |v| = scale (itself rounded twice) they
    differ by no more than 2 * 2^-8 (scale + |result|)."""
    d = (a.float() - b.float()).abs()
    assert (d <= 2.0 ** -7 * 1.02 * (scale.float() + b.float().abs())).all() and d.mean() <= 2e-3


# one token, edges of the 128-row tile and of the 256-row group, tails of a block, both block and head sizes
@pytest.mark.parametrize("tokens", [1, 2, 127, 128, 129, 187, 256, 300, 512])
@pytest.mark.parametrize("kind", ["plain", "strided", "heads_first", "wide", "broadcast"])
@pytest.mark.parametrize("call,head_dim,block,segment", [("dense", 128, 128, 512), ("dense", 64, 64, 512), ("dense", 64, 128, 512),
                                                          ("mean", 128, 128, 128), ("mean", 64, 64, 64)])
def test_in_place_equals_copied(tokens, kind, call, head_dim, block, segment):
    from pbs_attn_b200.prefill import MeanPooling_prefill, get_plan, permuted_block_sparse_attn_fwd
    w = Workload("inplace", 2, 4, 2, head_dim, tokens, "bf16", block, segment, 0.7, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=tokens, device="cuda")
    if kind == "broadcast":                     # a zero head stride: the copy is kept
        k, v = k[:, :1].expand(-1, 2, -1, -1), v[:, :1].expand(-1, 2, -1, -1)
    else:
        q, k, v = (_layout(t, kind) for t in (q, k, v))
    got, inters = [], []
    plan = get_plan(q, k.shape[1], block, segment)
    for impl, inter in (("tcgen05", None), ("tcgen05", {}), ("simt", {})):      # only calls without intermediates read in place
        if call == "mean":
            got.append(MeanPooling_prefill(q, k, v, block, segment, 0.7, attn_impl=impl, intermediates=inter))
        else:
            got.append(permuted_block_sparse_attn_fwd(q, k, v, block, segment, 0.7, True, attn_impl=impl, intermediates=inter))
        plan.check_status()
        inters.append((plan.key_indices.clone(), plan.block_mask.clone(), plan.first_block.clone()))
    assert all(torch.equal(a, b) for other in inters[1:] for a, b in zip(inters[0], other))
    assert torch.equal(got[0], got[1])
    if call == "mean":
        scale = MeanPooling_prefill(q, k, v.abs(), block, segment, 0.7, attn_impl="simt")
    else:
        scale = permuted_block_sparse_attn_fwd(q, k, v.abs(), block, segment, 0.7, True, attn_impl="simt")
    _same_but_for_rounding(got[0], got[2], scale)


# the result over K or V, whole or shifted by rows, and a second copy of the result over V
@pytest.mark.parametrize("tokens", [257, 300, 1000, 2048, 4096])
@pytest.mark.parametrize("where", ["k", "v", "v shifted", "replica on v"])
@pytest.mark.parametrize("call", ["dense", "mean"])
def test_result_may_overlap_keys_or_values(tokens, where, call):
    from pbs_attn_b200 import _cabi
    from pbs_attn_b200.prefill import Plan
    w = Workload("overlap", 1, 8, 8, 128, tokens, "bf16", 128, 128, 0.7, 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=tokens, device="cuda")
    plan = Plan(1, 8, 8, tokens, 128, 128, 4096 if call == "dense" else 128, q.dtype, q.device)
    kind = dict(no_permutation=True, diagonal_candidates=True) if call == "mean" else {}
    want = plan.run(q, k, v, torch.empty_like(q), plan.options(0.7, attn_impl="tcgen05", kv_in_place=True, **kind))
    buf = torch.empty(tokens + 64, 8, 128, dtype=q.dtype, device=q.device)       # (S, H, D) rows: a shift stays aligned
    seen = lambda t0: buf[t0 : t0 + tokens].transpose(0, 1)[None]
    shared = seen(64 if where == "v shifted" else 0).copy_(k if where == "k" else v)
    kk, vv = (shared, v) if where == "k" else (k, shared)
    out, reps = seen(0), None
    if where == "replica on v":
        out = torch.empty_like(seen(0))
        reps = _cabi.OutReplicas(1, 0, (_cabi.C.c_void_p * _cabi.MAX_OUT_REPLICAS)(shared.data_ptr()))
    plan.run(q, kk, vv, out, plan.options(0.7, attn_impl="tcgen05", out_replicas=reps, kv_in_place=True, **kind))
    torch.cuda.synchronize()
    plan.check_status()
    assert torch.equal(out, want)
    if reps is not None:
        assert torch.equal(seen(0), want)


@pytest.mark.parametrize("call", ["dense", "mean"])
def test_stages_after_a_call_work_on_its_keys_and_values(call):
    from pbs_attn_b200.prefill import MeanPooling_prefill, get_plan, permuted_block_sparse_attn_fwd, release_plans
    release_plans()
    block, segment, tokens = 128, (128 if call == "mean" else 512), 500
    fn = MeanPooling_prefill if call == "mean" else permuted_block_sparse_attn_fwd
    args = (block, segment, 0.7, True)
    inputs = [make_qkv(Workload("stages", 1, 4, 2, 128, tokens, "bf16", block, segment, 0.7, 5e5, sinks=4), seed=s, device="cuda")
              for s in (1, 2)]
    again = torch.empty_like(inputs[0][0])
    fn(*inputs[0], *args)                       # reads in place: nothing to go on with, and that is said
    plan = get_plan(inputs[0][0], 2, block, segment)
    with pytest.raises(RuntimeError, match="in place"):
        plan.attn_fwd(inputs[0][0], again)
    for q, k, v in inputs:
        inter = {}
        want = fn(q, k, v, *args, intermediates=inter)
        assert inter["plan"] is plan
        plan.attn_fwd(q, again, "simt")
        _same_but_for_rounding(again, want, fn(q, k, v.abs(), *args, attn_impl="simt"))
        fn(q, k, v, *args, intermediates=inter)
        assert torch.equal(plan.perm_k, k.repeat_interleave(2, dim=1)) and torch.equal(plan.perm_v, v.repeat_interleave(2, dim=1))
    fn(*inputs[0], *args)
    plan.segment_permute(inputs[0][1], inputs[0][2], identity=True)
    plan.attn_fwd(inputs[0][0], again)          # filled again
