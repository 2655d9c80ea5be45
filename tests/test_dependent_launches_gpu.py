"""Kernels that are set up while the one ahead of them still runs: chains in which every launch reads what the last one wrote,
writes what the last one read, or takes over memory that was just freed, against the same chain with a wait after each launch."""
import pytest

pytestmark = pytest.mark.gpu


def _chain(wait):
    import torch
    from scicompute_attention_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(11)
    bs, hq, hkv, d, blocks, seqs = 16, 8, 2, 128, 64, 3
    k, v = (torch.randn((blocks, bs, hkv, d), device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    table = torch.randperm(blocks, device="cuda", generator=g)[:seqs * 20].reshape(seqs, 20).to(torch.int32).contiguous()
    lens = torch.tensor([300, 17, 160], dtype=torch.int32, device="cuda")
    x = torch.randn((seqs, hq, 1, d), device="cuda", generator=g).to(torch.bfloat16)
    ids = torch.arange(seqs, dtype=torch.int32, device="cuda")
    kept = []

    def step(t):
        if wait:
            torch.cuda.synchronize()
        return t

    for i in range(40):
        new = step(x.view(seqs, hq, d)[:, :hkv].contiguous())
        step(ops.kv_append_batched(k, v, new, new, table, lens))               # reads the last output
        x = step(ops.paged_attention(x, k, v, table, lens, block_size=bs))      # reads the pool just written
        y = step(ops.flash_attention(x.view(1, hq, seqs, d), k[:1].view(1, hkv, bs, d), v[:1].view(1, hkv, bs, d)))
        x = step(ops.decode_attention(y.view(seqs, hq, 1, d), k[:seqs].view(seqs, hkv, bs, d), v[:seqs].view(seqs, hkv, bs, d)))
        z = step(ops.kv_gather(k, ids))
        step(ops.kv_append(k, v, z.view(-1, hkv, d)[:8], z.view(-1, hkv, d)[8:16], (lens.new_tensor([900 - i]) - torch.arange(8, device="cuda", dtype=torch.int32))))
        step(ops.kv_reset(k, v, ids[i % 3:i % 3 + 1]))
        f = step(ops.simt_attention(*(t.float() for t in (y, k[:1].view(1, hkv, bs, d), v[:1].view(1, hkv, bs, d)))))
        x = x + 0.25 * f.view(seqs, hq, 1, d).to(x.dtype) + torch.randn(x.shape, device="cuda", generator=g).to(x.dtype)
        del y, z, f, new
        if i % 10 == 9:
            kept += [x, k.clone(), v.clone()]
    torch.cuda.synchronize()
    return kept


def test_chains_without_waits_equal_chains_with_waits():
    import torch
    for a, b in zip(_chain(False), _chain(True)):
        assert torch.equal(a, b)


def test_captured_chain():
    import torch
    from scicompute_attention_b200 import ops
    q = torch.randn((1, 8, 40, 64), device="cuda").to(torch.float16)
    k, v = (torch.randn((1, 2, 300, 64), device="cuda").to(torch.float16) for _ in range(2))

    def chain(x):
        for _ in range(6):
            x = ops.flash_attention(x, k, v, causal=True)
            d = ops.decode_attention(x[:, :, :1].contiguous(), k, v)
            x = x + d
        return x
    expect = chain(q)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = chain(q)
    for _ in range(5):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, expect)
