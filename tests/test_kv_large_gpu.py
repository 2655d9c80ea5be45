"""KV append, reset and gather beyond one run of pieces per CTA, and beyond the pieces that 32 bits count, against plain indexing."""
import pytest

pytestmark = pytest.mark.gpu


def _check(blocks, bs, hkv, d, tokens, ids):
    import torch
    from scicompute_attention_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(d)
    k = torch.randint(-9000, 9000, (blocks, bs, hkv, d), device="cuda", generator=g, dtype=torch.int16)
    v = k.flip(0).contiguous()
    new = torch.randint(-9000, 9000, (tokens, hkv, d), device="cuda", generator=g, dtype=torch.int16)
    slots = torch.randperm(blocks * bs, device="cuda", generator=g)[:tokens].to(torch.int32)
    slots[::11] = -1
    ok = slots >= 0
    ek, ev = k.clone(), v.clone()
    ek.view(-1, hkv, d)[slots[ok].long()] = ev.view(-1, hkv, d)[slots[ok].long()] = new[ok]
    ops.kv_append(k, v, new, new, slots)
    assert torch.equal(k, ek) and torch.equal(v, ev)
    del new, ev
    out = ops.kv_gather(k, ids)
    _same_blocks(out, k, ids)
    ops.kv_reset(k, v, ids[:-1])
    keep = torch.ones(blocks, dtype=torch.bool, device="cuda")
    keep[ids[:-1].clamp(min=0).long()] = False
    assert torch.equal(k, ek * keep.view(-1, 1, 1, 1)) and not bool(v[~keep].any()) and bool(v[keep].any(dim=(1, 2, 3)).all())


def _same_blocks(out, pool, ids):
    import torch
    step = max(1, (1 << 30) // (pool[0].numel() * pool.element_size()))
    for at in range(0, len(ids), step):
        some = ids[at:at + step]
        want = pool[some.clamp(min=0).long()]
        want[some < 0] = 0
        assert torch.equal(out[at:at + step], want)


@pytest.mark.parametrize("hkv,d", ((8, 128), (3, 7)))  # pieces of 16 bytes, single bytes
def test_more_than_one_run_per_cta(hkv, d):
    import torch
    # a grid has 4736 CTAs (32 per SM) of 1024 pieces at most: 1.3 times that many pieces of each list
    piece, bs = (16, 16) if d == 128 else (1, 32)
    tokens = int(4736 * 1024 * 1.3) * piece // (hkv * d * 2)
    blocks = tokens // bs + 5
    ids = torch.randperm(blocks, device="cuda").to(torch.int32)
    ids[3] = -1
    _check(blocks, bs, hkv, d, tokens, ids)


def test_single_bytes_beyond_32_bits():
    import torch
    bs, hkv, d = 33, 31, 33  # a block of 67518 bytes: no multiple of 16
    blocks = 2**31 // (bs * hkv * d * 2) + 3
    ids = torch.randperm(blocks, device="cuda").to(torch.int32)
    _check(blocks, bs, hkv, d, 2**31 // (hkv * d * 2) + 2, ids)


def test_pieces_beyond_32_bits():
    import torch
    from scicompute_attention_b200 import ops
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 40 GB on the device")
    pool = torch.randint(-9000, 9000, (50, 256, 16, 128), device="cuda", dtype=torch.int16)  # blocks of 1 MB, 65536 pieces
    ids = torch.randint(-1, 50, (32771,), device="cuda", dtype=torch.int32)                   # 2^31 + 196608 pieces
    _same_blocks(ops.kv_gather(pool, ids), pool, ids)
