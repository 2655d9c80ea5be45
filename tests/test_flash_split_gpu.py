"""Prefill problems of so few query tiles that the CTAs of a cluster share the KV tiles of each (clusters of 2, 4 and 8), against
the FP64 oracle: dense, packed and paged, rows that see no key of some CTA's part, CTAs that get no tile at all."""
import numpy as np
import pytest

import helpers as H
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", (64, 96, 128, 256))
@pytest.mark.parametrize("dt", (ol.DT_F16, ol.DT_BF16))
def test_dense(dt, d):
    import torch
    from scicompute_attention_b200 import ops
    # tiles of 128 keys: 8 by 8, 9 of them by 8 (one CTA of eight gets one, three get none), 24; 40 items by 2; ragged ends
    for n, (b, hq, hkv, sq, skv, causal) in enumerate(((1, 2, 1, 100, 1024, True), (1, 4, 4, 1, 1100, True), (1, 2, 2, 130, 3000, False),
                                                       (5, 8, 2, 40, 901, True), (10, 4, 4, 128, 1029, True), (1, 1, 1, 700, 1300, True))):
        arrays = [H.uniform_inputs((b, h, s, d), 5000 + 3 * n + i, dt) for i, (h, s) in enumerate(((hq, sq), (hkv, skv), (hkv, skv)))]
        q, k, v = (H.to_device(bits, dt) for bits, _ in arrays)
        out, lse = ops.flash_attention(q, k, v, causal=causal, return_lse=True)
        torch.cuda.synchronize()
        expect, elog = ol.attention_f64(*(x for _, x in arrays), causal=causal, want_lse=True)
        H.check_close(H.to_host_f32(out), expect, dt, f"split D={d} case {n}")
        assert np.abs(lse.cpu().numpy() - elog).max() <= 1e-2
        again = ops.flash_attention(*(t.permute(0, 2, 1, 3).contiguous() for t in (q, k, v)), causal=causal, layout="bshd")
        assert torch.equal(again, out)


def test_what_is_not_a_number_stays_so():
    import torch
    from scicompute_attention_b200 import ops
    q, k, v = (torch.randn((1, 2, s, 128), device="cuda").to(torch.float16) for s in (64, 2000, 2000))
    clean = ops.flash_attention(q, k, v)
    q[0, 0, 7, 3] = float("nan")
    k[0, 1, 1500] = float("nan")  # a key of one CTA's part, seen by every row of head 1
    out = ops.flash_attention(q, k, v)
    assert bool(out[0, 0, 7].isnan().all()) and bool(out[0, 1].isnan().all())
    rest = [r for r in range(64) if r != 7]
    assert torch.equal(out[0, 0, rest], clean[0, 0, rest])


@pytest.mark.parametrize("d", (64, 128, 256))
def test_packed_equals_dense(d):
    import torch
    from scicompute_attention_b200 import ops
    lens = ((30, 1500), (1, 1100), (128, 1029))
    hq, hkv = 4, 2
    cu_q, cu_kv = (np.concatenate([[0], np.cumsum([x[i] for x in lens])]).astype(np.int32) for i in (0, 1))
    q, k, v = (torch.randn((n, h, d), device="cuda").to(torch.bfloat16) for n, h in ((cu_q[-1], hq), (cu_kv[-1], hkv), (cu_kv[-1], hkv)))
    out = ops.flash_attention_varlen(q, k, v, cu_q, cu_kv, causal=True)
    for s in range(len(lens)):
        rows, keys = slice(cu_q[s], cu_q[s + 1]), slice(cu_kv[s], cu_kv[s + 1])
        expect = ol.attention_f64(*(t.double().cpu().numpy().transpose(1, 0, 2)[None] for t in (q[rows], k[keys], v[keys])), causal=True)
        H.check_close(H.to_host_f32(out[rows]), expect[0].transpose(1, 0, 2), ol.DT_BF16, f"packed split D={d} sequence {s}")


@pytest.mark.parametrize("block", (8, 16, 64))
@pytest.mark.parametrize("d", (64, 128, 256))
def test_paged_with_a_part_of_unmapped_pages(d, block):
    import torch
    from scicompute_attention_b200 import ops
    n, m, hq, hkv = 1300, 20, 4, 2
    pages = -(-n // block)
    g = np.random.default_rng(8)
    table = g.permutation(pages + 3)[:pages].astype(np.int32)
    table[256 // block:640 // block] = -1  # all keys of one CTA's tiles
    kp, vp = (torch.randn((pages + 3, block, hkv, d), device="cuda").to(torch.float16) for _ in range(2))
    q = torch.randn((m, hq, d), device="cuda").to(torch.float16)
    out = ops.flash_attention_paged(q, kp, vp, torch.from_numpy(table[None]).cuda(), np.array([0, m], np.int32), np.array([n], np.int32), causal=True)
    torch.cuda.synchronize()
    keys = np.arange(n)
    mapped = table[keys // block] >= 0
    ks, vs = (t.double().cpu().numpy()[np.where(mapped, table[keys // block], 0), keys % block] for t in (kp, vp))
    score = np.einsum("thd,nhd->htn", q.double().cpu().numpy(), np.repeat(ks, hq // hkv, axis=1)) / np.sqrt(d)
    score = np.where((mapped[None, :] & (keys[None, :] <= np.arange(m)[:, None] + n - m))[None], score, -np.inf)
    w = np.exp(score - score.max(axis=-1, keepdims=True))
    expect = np.einsum("htn,nhd->thd", w / w.sum(axis=-1, keepdims=True), np.repeat(vs, hq // hkv, axis=1))
    H.check_close(H.to_host_f32(out), expect, ol.DT_F16, f"paged split D={d} block={block}")
