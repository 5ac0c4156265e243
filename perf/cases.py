"""Measured workloads of the prefill path, through the calls a program makes.

A case is a dict of plain values:
  call     "prefill"  permuted_block_sparse_attn_fwd on device tensors
           "mean"     MeanPooling_prefill (block selection without key permutation)
           "layer"    patched_attention_forward: projections, rotary embedding, prefill, output projection
           "host"     permuted_block_sparse_attn_fwd_host: pinned host tensors in, host tensor out
  batch, q_heads, kv_heads, head_dim, tokens, dtype, block, segment, threshold
  spread   standard deviation, over the (query block, key block) pairs, of the pooled block scores that is added to
           the nearly flat scores of pure noise.  0: a threshold t keeps about a share t of the causal blocks;
           above 0 the scores are log-normal, as attention with topics and recency is, and far fewer blocks are kept
  strided  True: q, k, v are (B, S, H, D) memory seen as (B, H, S, D), which is what a projection hands over
"""
import math
from functools import partial
from statistics import NormalDist

import torch

from pbs_attn_b200.hf_patch import patched_attention_forward
from pbs_attn_b200.prefill import (MeanPooling_prefill, permuted_block_sparse_attn_fwd,
                                   permuted_block_sparse_attn_fwd_host)
from pbs_attn_b200.synth import Workload, make_qkv, rope_tables

_DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_CHUNK = 512            # tokens that share a topic
_HIDDEN_PER_HEAD = 128  # model width per query head of the layer cases


def _case(name, call, batch, q_heads, kv_heads, head_dim, tokens, dtype="bf16", block=128, segment=256, threshold=0.9,
          spread=0.0, strided=False):
    return {"name": name, "call": call, "batch": batch, "q_heads": q_heads, "kv_heads": kv_heads, "head_dim": head_dim,
            "tokens": tokens, "dtype": dtype, "block": block, "segment": segment, "threshold": threshold,
            "spread": spread, "strided": strided}


def listed():
    return [
        # a short chat turn, below one segment: the dense fallback, where launches and host work are all there is
        _case("short_187", "prefill", 1, 32, 8, 128, 187, strided=True),
        # four prompts of ordinary length prefilled together
        _case("batch4_2k", "prefill", 4, 32, 8, 128, 2048, strided=True),
        # the fp32 configuration of the parity checks
        _case("fp32_2k", "prefill", 1, 4, 1, 64, 2048, dtype="fp32", block=64),
        # a ragged document in fp16 (tail shorter than a block, tail outside the last complete segment)
        _case("fp16_ragged_6k", "prefill", 1, 32, 8, 128, 6001, dtype="fp16", threshold=0.8, spread=1.0, strided=True),
        # 64-wide heads with 64-token blocks
        _case("head64_8k", "prefill", 1, 32, 8, 64, 8192, block=64, spread=1.0, strided=True),
        # one attention layer of a patched model: projections, rotary embedding, prefill, output projection
        _case("layer_8k", "layer", 1, 32, 8, 128, 8192),
        # block selection without permutation, at the defaults of the call
        _case("mean_16k", "mean", 1, 32, 8, 128, 16384, segment=1024, spread=1.0),
        # host tensors, copies pipelined with the computation
        _case("host_16k", "host", 1, 32, 8, 128, 16384),
        # 28 query heads on 4 KV heads, 64-token blocks in 512-token segments
        _case("block64_32k", "prefill", 1, 28, 4, 128, 32768, block=64, segment=512, strided=True),
        # a long document whose selection is sparse
        _case("sparse_32k", "prefill", 1, 32, 8, 128, 32768, spread=1.5, strided=True),
        # one rank's heads of an eight-way head-sharded call
        _case("rank_slice_128k", "prefill", 1, 4, 1, 128, 131072),
        # the benchmark's configuration
        _case("full_128k", "prefill", 1, 32, 8, 128, 131072),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["prefill"] * 6 + ["mean"] * 2 + ["layer"] * 2 + ["host"])
    dtype = rng.choice(["bf16"] * 6 + ["fp16"] * 2 + (["fp32"] if call in ("prefill", "mean") else []))
    q_heads, kv_heads, head_dim = rng.choice([(32, 8, 128), (32, 8, 128), (28, 4, 128), (4, 1, 128), (7, 1, 128), (32, 8, 64)])
    if dtype == "fp32":
        q_heads, kv_heads, head_dim = rng.choice([(4, 1, 64), (8, 2, 128)])
    block, segment = rng.choice([(128, 256), (128, 256), (128, 128), (128, 512), (64, 128), (64, 256), (64, 512), (128, 1024)])
    batch = rng.choice([1, 1, 1, 2, 4])
    lo, hi = {"prefill": (64, 131072), "mean": (256, 65536), "layer": (64, 32768), "host": (1024, 32768)}[call]
    # the work of a pass stays well below the largest listed case's (fp32 runs on the CUDA cores)
    most = 1.2e11 if dtype == "fp32" else 9e13
    hi = min(hi, int(math.sqrt(most / (2.0 * batch * q_heads * head_dim))))
    return {"call": call, "batch": batch, "q_heads": q_heads, "kv_heads": kv_heads, "head_dim": head_dim,
            "tokens": _log_int(rng, lo, hi), "dtype": dtype, "block": block, "segment": segment,
            "threshold": round(rng.uniform(0.5, 0.95), 3),
            "spread": round(rng.choice([0.0, rng.uniform(0.5, 2.0)]), 2) if call != "layer" else 0.0,
            "strided": call in ("prefill", "mean") and rng.random() < 0.6}


def _qkv(case, seed):
    dt = _DTYPE[case["dtype"]]
    w = Workload("case", case["batch"], case["q_heads"], case["kv_heads"], case["head_dim"], case["tokens"], case["dtype"],
                 case["block"], case["segment"], case["threshold"], 5e5, sinks=4)
    q, k, v = make_qkv(w, seed=seed, device="cuda")
    if case["spread"] > 0:
        # independent topic directions for queries and keys, constant over a chunk of tokens: the pooled score
        # of a block pair gets a normal part of standard deviation `spread`
        g = torch.Generator(device="cuda").manual_seed(seed + 1000003)
        for x in (q, k):
            n = -(-x.shape[2] // _CHUNK)
            t = torch.randn(*x.shape[:2], n, x.shape[3], generator=g, device="cuda") * math.sqrt(case["spread"])
            x += t.to(dt).repeat_interleave(_CHUNK, dim=2)[:, :, : x.shape[2]]
    return q, k, v


class _Attention(torch.nn.Module):
    """The parts of a decoder layer's attention that the patched forward uses."""

    def __init__(self, hidden, q_heads, kv_heads, head_dim, dtype, g):
        super().__init__()
        self.head_dim = head_dim
        self.layer_idx = 0
        for name, n_in, n_out in (("q_proj", hidden, q_heads * head_dim), ("k_proj", hidden, kv_heads * head_dim),
                                  ("v_proj", hidden, kv_heads * head_dim), ("o_proj", q_heads * head_dim, hidden)):
            lin = torch.nn.Linear(n_in, n_out, bias=False, device="cuda", dtype=dtype)
            lin.weight.data.copy_(torch.randn(n_out, n_in, generator=g, device="cuda") / math.sqrt(n_in))
            lin.weight.requires_grad_(False)
            setattr(self, name, lin)


def prepare(case, seed):
    if case["call"] == "layer":
        g = torch.Generator(device="cuda").manual_seed(seed)
        dt = _DTYPE[case["dtype"]]
        hidden = _HIDDEN_PER_HEAD * case["q_heads"]
        attn = _Attention(hidden, case["q_heads"], case["kv_heads"], case["head_dim"], dt, g)
        x = torch.randn(case["batch"], case["tokens"], hidden, generator=g, device="cuda").to(dt)
        cos, sin = rope_tables(case["tokens"], case["head_dim"], 5e5, "cuda")
        fn = partial(permuted_block_sparse_attn_fwd, block_size=case["block"], segment_size=case["segment"],
                     threshold=case["threshold"], causal=True)
        return {"case": case, "attn": attn, "x": x, "pos": (cos[None].to(dt), sin[None].to(dt)), "fn": fn}
    q, k, v = _qkv(case, seed)
    if case["call"] == "host":
        q, k, v = (t.cpu().pin_memory() for t in (q, k, v))
        return {"case": case, "q": q, "k": k, "v": v, "out": torch.empty_like(q).pin_memory()}
    if case["strided"]:
        q, k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v))
    return {"case": case, "q": q, "k": k, "v": v}


def run(state):
    c = state["case"]
    if c["call"] == "layer":
        with torch.no_grad():
            return patched_attention_forward(state["attn"], hidden_states=state["x"], position_embeddings=state["pos"],
                                             attention_mask=None, prefill_fn=state["fn"])[0]
    q, k, v = state["q"], state["k"], state["v"]
    if c["call"] == "mean":
        return MeanPooling_prefill(q, k, v, block_size=c["block"], segment_size=c["segment"], threshold=c["threshold"])
    if c["call"] == "host":
        return permuted_block_sparse_attn_fwd_host(q, k, v, c["block"], c["segment"], c["threshold"], out=state["out"])
    return permuted_block_sparse_attn_fwd(q, k, v, c["block"], c["segment"], c["threshold"], True)


def _kept_share(case):
    """Expected share of the causal triangle that the selection keeps."""
    seg = case["block"] if case["call"] == "mean" else case["segment"]
    own = min(1.0, seg / case["tokens"])                     # the query's own segment is always attended
    if case["spread"] > 0:
        n = NormalDist()
        share = 1.0 - n.cdf(case["spread"] - n.inv_cdf(case["threshold"]))
    else:
        share = case["threshold"]
    return min(1.0, own + (1.0 - own) * share)


def work(case):
    B, Hq, Hkv, S, D = (case[n] for n in ("batch", "q_heads", "kv_heads", "tokens", "head_dim"))
    e = 4 if case["dtype"] == "fp32" else 2
    bytes_ = (2 * Hq + 2 * Hkv) * B * S * D * e              # q, k, v read, the result written
    flops = 2.0 * B * Hq * D * S * S * _kept_share(case)     # Q K^T and P V over the kept part of the triangle
    if case["call"] == "prefill" and S > case["segment"]:
        flops += 2.0 * B * Hq * D * S * case["block"]        # key importance: the last block's logits
    if case["call"] == "layer":
        hidden = _HIDDEN_PER_HEAD * Hq
        flops += 2.0 * B * S * hidden * D * (2 * Hq + 2 * Hkv)
        # hidden states read and written, the weights read; q, k, v and the result live inside the call
        bytes_ = 2 * B * S * hidden * e + hidden * D * (2 * Hq + 2 * Hkv) * e + 2 * S * D * e
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # Measured by running the path against itself with head_dim (the hidden size, for a layer) in another order, and
    # against a float64 softmax over the same selection:
    #   fp32    8e-7, largest element 1.2e-5 (sums of up to 4000 terms)
    #   16-bit  2e-3 (bf16) and 3e-4 (fp16) from P and the result being 16-bit; where a pooled score or a key importance
    #           lands on its other 16-bit neighbour a query block attends another key block: up to 4.5e-3 in all, and
    #           a few rows differ by up to 0.75 of the root mean square
    #   layer   as above, but the 16-bit roundings of the projections move the selection of more blocks: 1.4e-2
    if case["dtype"] == "fp32":
        return {"rel": 4e-6, "max": 1e-4}
    return {"rel": 0.03 if case["call"] == "layer" else 0.015, "max": 0.99}


_EXACT_MOST = 7.2e10    # heads x tokens^2 that the 64-bit evaluation takes in about 20 seconds


def _exact_mask(q, k, case):
    """The selection for one query head: the permuted order of the keys and the block mask.

    Scores are summed in 64 bits and rounded to the input type where the path is defined to round them (after the dot
    product, after the division, and the pooled rows), because a block is kept or not by those rounded values."""
    S, D = q.shape
    bs, dt, f = case["block"], q.dtype, torch.float64
    mean = case["call"] == "mean"
    seg = bs if mean else case["segment"]
    rnd = lambda x: x.to(dt).to(f)
    idx = torch.arange(S, device=q.device)
    if not mean:
        L = S // seg * seg
        p = torch.softmax(rnd(rnd(q[-bs:].to(f) @ k[:L].to(f).T) / math.sqrt(D)), dim=-1).mean(dim=0)
        order = torch.sort(p.float().view(-1, seg), dim=-1, descending=True, stable=True).indices
        idx[:L] = (order + torch.arange(0, L, seg, device=q.device)[:, None]).flatten()
    nb = -(-S // bs)
    pool = lambda x: rnd(torch.nn.functional.pad(x.to(f), (0, 0, 0, nb * bs - S)).view(nb, bs, D).mean(dim=1))
    score = rnd(rnd(pool(q) @ pool(k[idx]).T) / math.sqrt(D))
    blk = torch.arange(nb, device=q.device)
    own = (blk[:, None] // (seg // bs)) == (blk // (seg // bs))
    cand = blk <= blk[:, None] if mean else (blk <= blk[:, None]) & ~own
    p = torch.nan_to_num(torch.softmax(score.masked_fill(~cand, -math.inf), dim=-1).float())
    val, order = torch.sort(p, dim=-1, descending=True, stable=True)
    reached = torch.cumsum(val.to(f), dim=-1).float() >= case["threshold"]
    keep = (blk <= reached.int().argmax(dim=-1, keepdim=True)) & reached.any(dim=-1, keepdim=True)
    mask = torch.zeros_like(keep).scatter(-1, order, keep) | own
    mask[:, int((idx == 0).nonzero()) // bs] = True
    return idx, mask


def _exact_attention(q, k, v, case):
    B, Hq, S, D = q.shape
    group = Hq // k.shape[1]
    out = torch.empty(B, Hq, S, D, dtype=torch.float64, device=q.device)
    bs = case["block"]
    seg = bs if case["call"] == "mean" else case["segment"]
    for b in range(B):
        for h in range(Hq):
            qh, kh, vh = q[b, h], k[b, h // group], v[b, h // group]
            pos = torch.arange(S, device=q.device)
            idx, mask = (pos, None) if case["call"] != "mean" and S <= seg else _exact_mask(qh, kh, case)
            kf, vf = kh[idx].double(), vh[idx].double()
            for r0 in range(0, S, 2048):
                r1 = min(r0 + 2048, S)
                n = S if mask is None else min(S, -(-r1 // seg) * seg)     # later segments are never attended
                s = qh[r0:r1].double() @ kf[:n].T
                s.mul_(1.0 / math.sqrt(D)).masked_fill_(idx[:n] > pos[r0:r1, None], -math.inf)
                if mask is not None:
                    s.masked_fill_(~mask[pos[r0:r1] // bs][:, pos[:n] // bs], -math.inf)
                out[b, h, r0:r1] = torch.softmax(s, dim=-1) @ vf[:n]
    return out


def exact(case, seed):
    """What run() returns, summed in 64 bits."""
    if case["batch"] * case["q_heads"] * case["tokens"] ** 2 > _EXACT_MOST:
        return None
    st = prepare(case, seed)
    if case["call"] == "layer":
        a, x = st["attn"], st["x"].double()
        B, S, _ = x.shape
        D, dt = case["head_dim"], st["x"].dtype
        cos, sin = (t.double()[:, None] for t in st["pos"])
        rnd = lambda t: t.to(dt).double()
        heads = lambda lin: rnd(x @ lin.weight.double().T).view(B, S, -1, D).transpose(1, 2)
        turn = lambda t: torch.cat((-t[..., D // 2:], t[..., :D // 2]), dim=-1)
        q, k = (rnd(rnd(t * cos) + rnd(turn(t) * sin)).to(dt) for t in (heads(a.q_proj), heads(a.k_proj)))
        o = rnd(_exact_attention(q, k, heads(a.v_proj).to(dt), case))
        return o.transpose(1, 2).reshape(B, S, -1) @ a.o_proj.weight.double().T
    return _exact_attention(*(st[n].cuda() for n in ("q", "k", "v")), case)
