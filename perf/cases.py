"""The attention work this library is used for, as cases that can be timed and compared.

A case is a plain dict; `listed()` names the ones that stand for the main uses, `draw(rng)` makes others of the same
ranges. `prepare(case, seed)` builds what a caller holds before the call (tensors on the GPU, page tables, host-side
length lists), `run(state)` is one pass through the public operators of `scicompute_attention_b200.ops`, and
`work(case)` counts what the pass cannot do without.

Kinds of case (field "kind"):
  prefill  ops.flash_attention          dense [B, H, S, D] prefill, causal or not, optionally with the log-sum-exp
  varlen   ops.flash_attention_varlen   prompts of a ragged batch, packed
  chunk    ops.flash_attention_paged    new tokens of every sequence against its paged KV cache
  decode   ops.decode_attention         one token per sequence against a contiguous KV cache
  step     ops.kv_append_batched + ops.paged_attention   one decode step of a paged batch
  cache    ops.kv_append, ops.kv_gather, ops.kv_reset    a prompt batch enters the pool, blocks are copied out and freed
  fp32     ops.simt_attention           the fp32 backend: reference-level results

Lengths of ragged batches are spread evenly over the case's range and dealt to the sequences in an order made from the
seed, so that the work of a case does not depend on the seed. Values are iid N(0, 1), cast to the case's type.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from scicompute_attention_b200 import ops

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}

# No drawn case does more than the largest listed ones: FLOPs of the four-prompt prefill, bytes of the 256-sequence step.
MOST_FLOPS = 5.5e11
MOST_BYTES = 4.5e9


def listed():
    layer = {"heads": 32, "kv_heads": 8, "head_dim": 128, "dtype": "bf16"}
    return [
        # a short prompt of one chat turn: the whole prefill is a few microseconds of GPU work
        dict(layer, name="prefill_one_short_prompt", kind="prefill", batch=1, seq_q=203, seq_kv=203, causal=True,
             lse=False, layout="bhsd"),
        # four prompts of 4096 tokens, one layer of a 32 / 8 head model: the throughput-bound prefill
        dict(layer, name="prefill_four_long_prompts", kind="prefill", batch=4, seq_q=4096, seq_kv=4096, causal=True,
             lse=False, layout="bhsd"),
        # bidirectional attention with small heads, activations as [B, S, H, D], log-sum-exp kept for a later merge
        {"name": "prefill_d64_bidirectional_lse", "kind": "prefill", "batch": 3, "heads": 32, "kv_heads": 8,
         "head_dim": 64, "dtype": "fp16", "seq_q": 2900, "seq_kv": 2900, "causal": False, "lse": True, "layout": "bshd"},
        # wide heads: one prompt
        {"name": "prefill_d256_prompt", "kind": "prefill", "batch": 1, "heads": 32, "kv_heads": 8, "head_dim": 256,
         "dtype": "bf16", "seq_q": 3000, "seq_kv": 3000, "causal": True, "lse": False, "layout": "bhsd"},
        # the prompts of a rollout batch, packed without padding
        dict(layer, name="varlen_rollout_prompts", kind="varlen", seqs=10, min_len=64, max_len=4096, causal=True),
        # follow-up prompts: a few hundred new tokens per sequence against the cache of the conversation so far
        dict(layer, name="chunk_follow_up_prompts", kind="chunk", seqs=20, min_new=16, max_new=500, min_len=512,
             max_len=6000, block_size=16),
        # one user, short context: the latency of a single decode call
        dict(layer, name="decode_one_sequence", kind="decode", batch=1, seq_kv=1000, ragged=False),
        # 128 sequences of 4096 tokens: the bandwidth-bound decode
        dict(layer, name="decode_128_sequences", kind="decode", batch=128, seq_kv=4096, ragged=False),
        # a handful of short conversations in a paged cache
        dict(layer, name="step_few_sequences", kind="step", seqs=6, min_len=33, max_len=900, block_size=16),
        # a full server: 256 sequences of 512 to 8192 tokens scattered over the pool
        dict(layer, name="step_256_sequences", kind="step", seqs=256, min_len=512, max_len=8192, block_size=16),
        # a prompt batch is written to the pool, blocks are copied out (swap, prefix export), others are freed
        dict(layer, name="cache_fill_copy_free", kind="cache", seqs=24, min_len=64, max_len=4096, block_size=16,
             gather=1500, reset=1000),
        # the fp32 backend on the shape the results of the other backends are checked on
        {"name": "fp32_reference_forward", "kind": "fp32", "batch": 1, "heads": 8, "kv_heads": 8, "head_dim": 128,
         "dtype": "fp32", "seq_q": 1024, "seq_kv": 1024, "causal": False, "lse": False, "layout": "bhsd"},
    ]


# ------------------------------------------------------------------------------------------------
# drawn cases
# ------------------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _layer(rng, dims=(64, 128, 128, 128, 256)):
    heads, kv_heads = rng.choice([(32, 8), (32, 8), (32, 8), (8, 8), (16, 2), (6, 3)])
    return {"heads": heads, "kv_heads": kv_heads, "head_dim": rng.choice(dims), "dtype": rng.choice(["bf16", "bf16", "fp16"])}


def _fits(case, flops=MOST_FLOPS, nbytes=MOST_BYTES):
    w = work(case)
    return w["flops"] <= flops and w["bytes"] <= nbytes


def draw(rng):
    while True:
        case = _draw(rng)
        if case["kind"] == "fp32":
            if _fits(case, flops=4.3e9):
                return case
        elif _fits(case):
            return case


def _draw(rng):
    kind = rng.choice(["prefill"] * 4 + ["varlen", "chunk", "decode", "decode", "step", "step", "cache", "fp32"])
    if kind == "prefill":
        skv = _log(rng, 16, 6000)
        sq = skv if rng.random() < 0.75 else max(1, int(skv * rng.uniform(0.05, 1.0)))
        return dict(_layer(rng), kind=kind, batch=_log(rng, 1, 8), seq_q=sq, seq_kv=skv, causal=rng.random() < 0.7,
                    lse=rng.random() < 0.25, layout=rng.choice(["bhsd", "bshd"]))
    if kind == "varlen":
        lo = _log(rng, 8, 600)
        return dict(_layer(rng), kind=kind, seqs=_log(rng, 2, 64), min_len=lo, max_len=lo + _log(rng, 8, 4096),
                    causal=rng.random() < 0.8)
    if kind == "chunk":
        new, lo = _log(rng, 1, 200), _log(rng, 64, 2000)
        most_new = new + _log(rng, 4, 600)
        return dict(_layer(rng), kind=kind, seqs=_log(rng, 1, 48), min_new=new, max_new=most_new, min_len=lo + most_new,
                    max_len=lo + most_new + _log(rng, 32, 8000), block_size=rng.choice([16, 16, 32]))
    if kind == "decode":
        return dict(_layer(rng), kind=kind, batch=_log(rng, 1, 128), seq_kv=_log(rng, 50, 131072), ragged=rng.random() < 0.4)
    if kind == "step":
        lo = _log(rng, 16, 1000)
        return dict(_layer(rng), kind=kind, seqs=_log(rng, 1, 256), min_len=lo, max_len=lo + _log(rng, 32, 8192),
                    block_size=rng.choice([16, 16, 16, 32]))
    if kind == "cache":
        lo = _log(rng, 16, 500)
        return dict(_layer(rng), kind=kind, seqs=_log(rng, 1, 64), min_len=lo, max_len=lo + _log(rng, 32, 6000),
                    block_size=rng.choice([16, 16, 32]), gather=_log(rng, 8, 4000), reset=_log(rng, 8, 4000))
    heads, kv_heads = rng.choice([(8, 8), (8, 2), (16, 4)])
    s = _log(rng, 40, 1300)
    return {"kind": kind, "batch": _log(rng, 1, 4), "heads": heads, "kv_heads": kv_heads,
            "head_dim": rng.choice([64, 128]), "dtype": "fp32", "seq_q": s, "seq_kv": s, "causal": rng.random() < 0.5,
            "lse": rng.random() < 0.25, "layout": "bhsd"}


# ------------------------------------------------------------------------------------------------
# sizes that follow from a case
# ------------------------------------------------------------------------------------------------
def _spread(lo, hi, n):
    """n whole lengths, evenly over [lo, hi]."""
    return [(lo + hi) // 2] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _lengths(case):
    """(query tokens, keys) of every sequence of a ragged case."""
    if case["kind"] == "chunk":
        new, total = _spread(case["min_new"], case["max_new"], case["seqs"]), _spread(case["min_len"], case["max_len"], case["seqs"])
        return list(zip(new, total))
    if case["kind"] == "decode":
        n = case["seq_kv"]
        return [(1, x) for x in (_spread(max(1, n // 4), n, case["batch"]) if case["ragged"] else [n] * case["batch"])]
    return [(1 if case["kind"] == "step" else x, x) for x in _spread(case["min_len"], case["max_len"], case["seqs"])]


def _blocks(case, lens):
    return [-(-n // case["block_size"]) for n in lens]


def work(case):
    """Bytes: every input read once, every output written once. FLOPs: 4 * D for every visible (query, key) pair."""
    hq, hkv, d, e = case["heads"], case["kv_heads"], case["head_dim"], BYTES[case["dtype"]]
    kind = case["kind"]
    if kind in ("prefill", "fp32"):
        b, sq, skv = case["batch"], case["seq_q"], case["seq_kv"]
        pairs = sq * skv - (sq * (sq - 1) // 2 if case["causal"] else 0)  # query i of the last sq sees skv - sq + i + 1 keys
        nbytes = e * d * b * (2 * hq * sq + 2 * hkv * skv) + (4 * b * hq * sq if case["lse"] else 0)
        return {"bytes": nbytes, "flops": 4 * b * hq * d * pairs}
    if kind == "cache":
        tokens = sum(n for _, n in _lengths(case))
        block = case["block_size"] * hkv * d * e
        copied, freed = 2 * case["gather"] * block, case["reset"] * block  # K and V blocks copied out; freed ones per pool
        return {"bytes": 4 * tokens * hkv * d * e + 4 * tokens + 2 * copied + 2 * freed + 4 * (2 * case["gather"] + case["reset"]), "flops": 0}
    lens = _lengths(case)
    rows, keys = sum(q for q, _ in lens), sum(n for _, n in lens)
    causal = kind == "chunk" or case.get("causal", False)
    pairs = sum(q * n - (q * (q - 1) // 2 if causal else 0) for q, n in lens)
    nbytes = e * d * (2 * hq * rows + 2 * hkv * keys)
    if kind in ("chunk", "step"):
        nbytes += 4 * sum(_blocks(case, [n for _, n in lens])) + 4 * len(lens)
    if kind == "step":
        nbytes += 2 * len(lens) * hkv * d * e  # the new tokens are read once more when they are appended
    return {"bytes": nbytes, "flops": 4 * hq * d * pairs}


def tolerance(case):
    """About four times the distance of the results from the same attention in 64 bits. Measured 2-norms: bf16 1.7e-3
    (the rounding of the output), fp16 3e-4, fp32 8e-7; largest differences: 6e-3, 3e-3, 4e-6. Moved bytes stay the same."""
    if case["kind"] == "cache":
        return "exact"
    return {"rel": {"bf16": 7e-3, "fp16": 1.2e-3, "fp32": 4e-6}[case["dtype"]], "max": {"bf16": 2.5e-2, "fp16": 1.2e-2, "fp32": 3e-5}[case["dtype"]]}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _randn(gen, case, *shape):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).to(DTYPES[case["dtype"]])


def _pool(gen, case, blocks):
    """K or V pool of a paged cache, filled in pieces (the fp32 numbers of a large one would not fit)."""
    shape = (blocks, case["block_size"], case["kv_heads"], case["head_dim"])
    pool = torch.empty(shape, device="cuda", dtype=DTYPES[case["dtype"]])
    for at in range(0, blocks, 8192):
        piece = pool[at:at + 8192]
        piece.copy_(torch.randn(piece.shape, generator=gen, device="cuda", dtype=torch.float32))
    return pool


def _table(gen, counts, pool_blocks):
    """int32 page table [sequences, longest], blocks dealt from a shuffled pool; -1 behind a sequence's last block."""
    ids = torch.randperm(pool_blocks, generator=gen, device="cuda").to(torch.int32)
    n = torch.tensor(counts, device="cuda")
    first = torch.cumsum(n, 0) - n
    col = torch.arange(max(counts), device="cuda")
    at = first[:, None] + col[None, :]
    table = torch.where(col[None, :] < n[:, None], ids[at.clamp(max=pool_blocks - 1)], torch.full_like(at, -1, dtype=torch.int32))
    return table.contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    order = np.random.default_rng(seed)
    hq, hkv, d = case["heads"], case["kv_heads"], case["head_dim"]
    kind = case["kind"]
    s = {"case": case}
    if kind in ("prefill", "fp32"):
        b, sq, skv = case["batch"], case["seq_q"], case["seq_kv"]
        shape = (lambda h, n: (b, h, n, d)) if case["layout"] == "bhsd" else (lambda h, n: (b, n, h, d))
        s["q"], s["k"], s["v"] = _randn(gen, case, *shape(hq, sq)), _randn(gen, case, *shape(hkv, skv)), _randn(gen, case, *shape(hkv, skv))
        return s

    lens = _lengths(case)
    lens = [lens[i] for i in order.permutation(len(lens))]
    rows, keys = [q for q, _ in lens], [n for _, n in lens]
    if kind == "varlen":
        total = sum(keys)
        s["q"], s["k"], s["v"] = _randn(gen, case, total, hq, d), _randn(gen, case, total, hkv, d), _randn(gen, case, total, hkv, d)
        s["cu"] = np.concatenate([[0], np.cumsum(keys)]).astype(np.int32)
        return s
    if kind == "decode":
        b, n = case["batch"], case["seq_kv"]
        s["q"], s["k"], s["v"] = _randn(gen, case, b, hq, 1, d), _pool_like(gen, case, b, hkv, n, d), _pool_like(gen, case, b, hkv, n, d)
        s["lens"] = torch.tensor(keys, dtype=torch.int32, device="cuda") if case["ragged"] else None
        return s

    counts = _blocks(case, keys)
    blocks = sum(counts) + sum(counts) // 8 + 16  # the pool is never quite full
    if kind == "cache":
        blocks += case["gather"] + case["reset"]
    s["k_pool"], s["v_pool"] = _pool(gen, case, blocks), _pool(gen, case, blocks)
    if kind == "cache":
        ids = torch.randperm(blocks, generator=gen, device="cuda").to(torch.int32)
        used = sum(counts)
        s["gather"], s["reset"] = ids[used:used + case["gather"]].contiguous(), ids[used + case["gather"]:used + case["gather"] + case["reset"]].contiguous()
        bs, slots, at = case["block_size"], [], 0
        for n, c in zip(keys, counts):
            t = torch.arange(n, device="cuda")
            slots.append(ids[at + t // bs] * bs + (t % bs).to(torch.int32))
            at += c
        s["slots"] = torch.cat(slots).to(torch.int32)
        s["k_new"], s["v_new"] = _randn(gen, case, sum(keys), hkv, d), _randn(gen, case, sum(keys), hkv, d)
        return s
    s["table"] = _table(gen, counts, blocks)
    if kind == "chunk":
        s["q"] = _randn(gen, case, sum(rows), hq, d)
        s["cu"], s["lens"] = np.concatenate([[0], np.cumsum(rows)]).astype(np.int32), np.array(keys, dtype=np.int32)
        return s
    s["q"] = _randn(gen, case, len(keys), hq, 1, d)
    s["k_new"], s["v_new"] = _randn(gen, case, len(keys), hkv, d), _randn(gen, case, len(keys), hkv, d)
    s["lens"] = torch.tensor(keys, dtype=torch.int32, device="cuda")  # the new token included
    s["mean"], s["longest"] = sum(keys) // len(keys), max(keys)
    return s


def _pool_like(gen, case, b, h, n, d):
    out = torch.empty((b, h, n, d), device="cuda", dtype=DTYPES[case["dtype"]])
    for i in range(b):
        out[i].copy_(torch.randn((h, n, d), generator=gen, device="cuda", dtype=torch.float32))
    return out


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "prefill":
        return ops.flash_attention(s["q"], s["k"], s["v"], causal=case["causal"], return_lse=case["lse"], layout=case["layout"])
    if kind == "varlen":
        return ops.flash_attention_varlen(s["q"], s["k"], s["v"], s["cu"], s["cu"], causal=case["causal"])
    if kind == "chunk":
        return ops.flash_attention_paged(s["q"], s["k_pool"], s["v_pool"], s["table"], s["cu"], s["lens"], causal=True)
    if kind == "decode":
        return ops.decode_attention(s["q"], s["k"], s["v"], seq_lens=s["lens"])
    if kind == "step":
        ops.kv_append_batched(s["k_pool"], s["v_pool"], s["k_new"], s["v_new"], s["table"], s["lens"])
        out = ops.paged_attention(s["q"], s["k_pool"], s["v_pool"], s["table"], s["lens"], block_size=case["block_size"],
                                  typical_len=s["mean"], longest_len=s["longest"])
        return out, s["k_pool"], s["v_pool"]
    if kind == "cache":
        ops.kv_append(s["k_pool"], s["v_pool"], s["k_new"], s["v_new"], s["slots"])
        copied = ops.kv_gather(s["k_pool"], s["gather"]), ops.kv_gather(s["v_pool"], s["gather"])
        ops.kv_reset(s["k_pool"], s["v_pool"], s["reset"])
        return (*copied, s["k_pool"], s["v_pool"])
    return ops.simt_attention(s["q"], s["k"], s["v"], causal=case["causal"], return_lse=case["lse"], layout=case["layout"])
