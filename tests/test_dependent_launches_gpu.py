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


@pytest.mark.parametrize("hkv,d", ((8, 128), (3, 7)))  # a token of 16-byte pieces, of single bytes
def test_a_kernel_that_writes_for_long_and_the_one_that_reads_it(hkv, d):
    """The writer runs for many times what it takes to set the reader up, so the reader is there from the writer's first CTAs on."""
    import torch
    from scicompute_attention_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(d)
    bs, blocks = 16, 3000
    k, v = (torch.zeros((blocks, bs, hkv, d), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    slots = torch.randperm(blocks * bs, device="cuda", generator=g).to(torch.int32)
    ids = torch.randperm(blocks, device="cuda", generator=g).to(torch.int32)
    new = [tuple(torch.randn((blocks * bs, hkv, d), device="cuda", generator=g).to(torch.bfloat16) for _ in range(2)) for _ in range(3)]
    got = []
    for kn, vn in new:
        ops.kv_append(k, v, kn, vn, slots)
        got.append((ops.kv_gather(k, ids), ops.kv_gather(v, ids)))
        copied = got[-1][0]
        ops.kv_append(k, v, copied.view(-1, hkv, d), got[-1][1].view(-1, hkv, d), slots)  # what was just copied out goes in again
        ops.kv_reset(k, v, ids[:blocks // 2])
        got.append((ops.kv_gather(k, ids), ops.kv_gather(v, ids)))
    for i, pair in enumerate(new):
        for j, n in enumerate(pair):
            pool = torch.empty_like(k)
            pool.view(-1, hkv, d)[slots.long()] = n
            out = pool[ids.long()]
            assert torch.equal(got[2 * i][j], out)
            pool.view(-1, hkv, d)[slots.long()] = out.view(-1, hkv, d)
            pool[ids[:blocks // 2].long()] = 0
            assert torch.equal(got[2 * i + 1][j], pool[ids.long()])


def test_an_append_and_the_attention_over_it():
    import torch
    from scicompute_attention_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(5)
    bs, hq, hkv, d, seqs, pages = 16, 8, 2, 128, 64, 64
    k, v = (torch.zeros((seqs * pages, bs, hkv, d), device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.randperm(seqs * pages, device="cuda", generator=g).to(torch.int32).view(seqs, pages).contiguous()
    lens = torch.full((seqs,), pages * bs, dtype=torch.int32, device="cuda")
    at = (table.long()[:, :, None] * bs + torch.arange(bs, device="cuda")).view(-1).to(torch.int32)
    q = torch.randn((seqs, hq, 1, d), device="cuda", generator=g).to(torch.bfloat16)
    new = [tuple(torch.randn((seqs * pages * bs, hkv, d), device="cuda", generator=g).to(torch.bfloat16) for _ in range(2)) for _ in range(4)]
    got = []
    for kn, vn in new:
        ops.kv_append(k, v, kn, vn, at)
        got.append(ops.paged_attention(q, k, v, table, lens, block_size=bs))
    for (kn, vn), out in zip(new, got):
        dense = (t.view(seqs, pages * bs, hkv, d).permute(0, 2, 1, 3).contiguous() for t in (kn, vn))
        want = torch.nn.functional.scaled_dot_product_attention(q.float(), *(t.float() for t in dense), enable_gqa=True)
        assert float((out.float() - want).norm() / want.norm()) < 4e-3  # the rounding of a bf16 output is 1.7e-3


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
