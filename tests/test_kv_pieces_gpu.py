"""KV append, reset and gather at the edges of a CTA's run of pieces, in 16-byte pieces and byte by byte, with slots and blocks
that are to be left out, against plain indexing."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,dtype", ((8, "float16"), (128, "bfloat16"), (7, "float16")))  # a token of 2 pieces, of 32, of 28 bytes
@pytest.mark.parametrize("tokens", (1, 31, 32, 33, 255, 512, 513, 4000))
def test_append_reset_gather(tokens, d, dtype):
    import torch
    from scicompute_attention_b200 import ops
    bs, hkv, blocks = 16, 2, 300
    g = torch.Generator(device="cuda").manual_seed(tokens * 10 + d)
    k, v = (torch.randn((blocks, bs, hkv, d), device="cuda", generator=g).to(getattr(torch, dtype)) for _ in range(2))
    kn, vn = (torch.randn((tokens, hkv, d), device="cuda", generator=g).to(k.dtype) for _ in range(2))
    slots = torch.randperm(blocks * bs, device="cuda", generator=g)[:tokens].to(torch.int32)
    slots[::7] = -1                      # not stored
    slots[3::50] = blocks * bs + 5       # beyond the pool: not stored
    ek, ev = k.clone(), v.clone()
    ok = (slots >= 0) & (slots < blocks * bs)
    ek.view(-1, hkv, d)[slots[ok].long()], ev.view(-1, hkv, d)[slots[ok].long()] = kn[ok], vn[ok]
    ops.kv_append(k, v, kn, vn, slots)
    assert torch.equal(k, ek) and torch.equal(v, ev)
    ids = torch.randperm(blocks, device="cuda", generator=g)[:min(blocks, max(1, tokens // 8))].to(torch.int32)
    ids[2::5] = -1
    out = ops.kv_gather(k, ids)
    assert torch.equal(out, torch.where((ids >= 0)[:, None, None, None], k[ids.clamp(min=0).long()], torch.zeros_like(out)))
    ops.kv_reset(k, v, ids)
    ek[ids[ids >= 0].long()], ev[ids[ids >= 0].long()] = 0, 0
    assert torch.equal(k, ek) and torch.equal(v, ev)
