"""Prefill geometries whose P has tensor-memory columns of its own (head dims up to 64 and above 128; at D=256 a KV tile takes
two ring slots): key counts around the edges of one to three KV tiles, one and two query tiles per item, several items per
CTA, dense and over a paged cache with unmapped pages, against the FP64 oracle."""
import numpy as np
import pytest

import helpers as H
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", (32, 64, 160, 256))
@pytest.mark.parametrize("dt", (ol.DT_F16, ol.DT_BF16))
def test_key_counts_around_tile_edges(dt, d):
    import torch
    from scicompute_attention_b200 import ops
    for n, (sq, skv) in enumerate(((1, 1), (3, 64), (64, 65), (127, 127), (128, 128), (129, 129), (60, 255), (130, 257), (300, 385))):
        for causal in (False, True):
            arrays = [H.uniform_inputs((1, h, s, d), 900 + 3 * n + i, dt) for i, (h, s) in enumerate(((4, sq), (2, skv), (2, skv)))]
            q, k, v = (H.to_device(bits, dt) for bits, _ in arrays)
            out = ops.flash_attention(q, k, v, causal=causal)
            torch.cuda.synchronize()
            expect = ol.attention_f64(*(x for _, x in arrays), causal=causal)
            H.check_close(H.to_host_f32(out), expect, dt, f"D={d} Sq={sq} Skv={skv} causal={causal}")


@pytest.mark.parametrize("d", (64, 256))
def test_many_items_per_cta(d):
    """600 items on the 148 SMs: every barrier goes through several items; each batch element repeats the first one's bits."""
    import torch
    from scicompute_attention_b200 import ops
    b, h, s = 75, 8, 300
    q, k, v = (torch.randn((1, h, s, d), device="cuda", dtype=torch.float32).to(torch.bfloat16).expand(b, h, s, d).contiguous() for _ in range(3))
    out = ops.flash_attention(q, k, v, causal=True)
    torch.cuda.synchronize()
    assert torch.equal(out, out[:1].expand_as(out))
    expect = ol.attention_f64(*(t[:1].double().cpu().numpy() for t in (q, k, v)), causal=True)
    H.check_close(H.to_host_f32(out[:1]), expect, ol.DT_BF16, f"D={d}")


@pytest.mark.parametrize("block", (8, 16, 64))
@pytest.mark.parametrize("d", (64, 256))
def test_paged_with_unmapped_pages(d, block):
    import torch
    from scicompute_attention_b200 import ops
    rng = np.random.default_rng(5)
    hq, hkv, lens, new = 4, 2, (257, 130, 64), (40, 130, 1)
    pages = [-(-n // block) for n in lens]
    pool = sum(pages) + 3
    ids = rng.permutation(pool)
    table = np.full((3, max(pages)), -1, np.int32)
    at = 0
    for s, n in enumerate(pages):
        table[s, :n] = ids[at:at + n]
        at += n
    holes = [(0, pages[0] // 2)]  # a page in the middle of the longest sequence: its keys have no weight
    for s, p in holes:
        table[s, p] = -1
    kp, vp = (torch.randn((pool, block, hkv, d), device="cuda").to(torch.float16) for _ in range(2))
    q = torch.randn((sum(new), hq, d), device="cuda").to(torch.float16)
    cu = np.concatenate([[0], np.cumsum(new)]).astype(np.int32)
    out = ops.flash_attention_paged(q, kp, vp, torch.from_numpy(table).cuda(), cu, np.array(lens, np.int32), causal=True)
    torch.cuda.synchronize()
    for s, (n, m) in enumerate(zip(lens, new)):
        keys = np.arange(n)
        mapped = table[s][keys // block] >= 0
        row = np.where(mapped, table[s][keys // block], 0)
        ks, vs = (t.float().cpu().numpy()[row, keys % block].astype(np.float64) for t in (kp, vp))  # [n, hkv, d]
        qs = q[cu[s]:cu[s + 1]].double().cpu().numpy()
        score = np.einsum("thd,nhd->htn", qs, np.repeat(ks, hq // hkv, axis=1)) / np.sqrt(d)
        seen = mapped[None, :] & (keys[None, :] <= np.arange(m)[:, None] + n - m)
        score = np.where(seen[None], score, -np.inf)
        w = np.exp(score - score.max(axis=-1, keepdims=True))
        w /= w.sum(axis=-1, keepdims=True)
        expect = np.einsum("htn,nhd->thd", w, np.repeat(vs, hq // hkv, axis=1))
        H.check_close(H.to_host_f32(out[cu[s]:cu[s + 1]]), expect, ol.DT_F16, f"paged D={d} block={block} sequence {s}")
