"""Decode calls small enough for the one-launch cluster kernel, at the edges of its range, against the FP64 oracle."""
import ctypes as C

import numpy as np
import pytest

import helpers as H
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,batch,hq,hkv,skv,d,cluster", [
    (ol.DT_BF16, 1, 8, 8, 1, 128, (8,)),       # one key: seven CTAs of every cluster hold nothing
    (ol.DT_F16, 1, 4, 1, 449, 64, (8,)),       # 8 steps for 8 CTAs, the last one with a single key
    (ol.DT_BF16, 1, 32, 8, 1000, 128, (8,)),
    (ol.DT_BF16, 6, 32, 8, 900, 128, (4,)),
    (ol.DT_F16, 16, 32, 8, 500, 128, (2,)),
    (ol.DT_BF16, 2, 32, 1, 700, 128, (8,)),    # two head chunks of 16 query heads
    (ol.DT_F16, 1, 12, 1, 130, 96, (8,)),      # 12 heads: both row halves, one of them ragged
    (ol.DT_BF16, 2, 8, 8, 300, 256, (4, 8)),   # one CTA per SM: 16 clusters of 8 fit or not, by the SMs per GPC
])
def test_cluster_decode_matches_the_oracle(dt, batch, hq, hkv, skv, d, cluster):
    import torch
    from scicompute_attention_b200 import ops
    qb, qd = H.normal_inputs((batch, hq, 1, d), 74000, dt)
    kb, kd = H.normal_inputs((batch, hkv, skv, d), 74001, dt)
    vb, vd = H.uniform_inputs((batch, hkv, skv, d), 74002, dt)
    q, k, v = H.to_device(qb, dt), H.to_device(kb, dt), H.to_device(vb, dt)
    out, stats = ops.decode_attention(q, k, v, return_stats=True)
    assert stats["cluster"] in cluster
    H.check_close(H.to_host_f32(out), ol.attention_f64(qd, kd, vd, causal=True), dt)
    # ragged, an empty sequence among them: its rows are zero
    lens = np.array([(skv * (i + 1)) // batch for i in range(batch)], dtype=np.int32)
    lens[-1] = 0
    out, stats = ops.decode_attention(q, k, v, seq_lens=torch.from_numpy(lens).cuda(), return_stats=True)
    assert stats["cluster"] > 0
    out = H.to_host_f32(out)
    for b, n in enumerate(lens):
        if n == 0:
            assert (out[b] == 0).all()
        else:
            H.check_close(out[b:b + 1], ol.attention_f64(qd[b:b + 1], kd[b:b + 1, :, :n], vd[b:b + 1, :, :n], causal=True), dt)


@pytest.mark.parametrize("block_size,seqs,longest", [(16, 1, 700), (8, 5, 333), (32, 16, 400)])
def test_cluster_paged_decode_with_holes(block_size, seqs, longest):
    import torch
    from scicompute_attention_b200 import ops
    dt, hq, hkv, d = ol.DT_BF16, 8, 4, 128
    width = -(-longest // block_size)
    rng = np.random.default_rng(3)
    pool = seqs * width + 5
    table = rng.permutation(pool)[:seqs * width].astype(np.int32).reshape(seqs, width)
    table[0, width // 2] = -1
    lens = np.linspace(1, longest, seqs).astype(np.int32) if seqs > 1 else np.array([longest], np.int32)
    qb, qd = H.normal_inputs((seqs, hq, 1, d), 75000, dt)
    kb, kd = H.normal_inputs((pool, block_size, hkv, d), 75001, dt)
    vb, vd = H.uniform_inputs((pool, block_size, hkv, d), 75002, dt)
    out, stats = ops.paged_attention(H.to_device(qb, dt), H.to_device(kb, dt), H.to_device(vb, dt), torch.from_numpy(table).cuda(),
                                     torch.from_numpy(lens).cuda(), block_size=block_size, return_stats=True)
    assert stats["cluster"] > 0
    expect = ol.paged_decode_f64(qd[:, :, 0], kd, vd, table, lens, block_size)
    H.check_close(H.to_host_f32(out), expect.reshape(seqs, hq, 1, d), dt)


@pytest.mark.parametrize("batch,hq,hkv,skv,d", [
    (2, 8, 8, 4000, 256),    # 24.2 us on clusters of 4, 20.5 with the schedule
    (16, 16, 1, 4000, 256),  # 32.8 / 24.5
    (16, 8, 8, 16000, 64),   # 86.1 / 81.5
])
def test_calls_that_the_schedule_does_faster_stay_with_it(batch, hq, hkv, skv, d):
    import torch
    from scicompute_attention_b200 import ops
    q = torch.zeros(batch, hq, 1, d, device="cuda", dtype=torch.bfloat16)
    k = torch.zeros(batch, hkv, skv, d, device="cuda", dtype=torch.bfloat16)
    assert ops.decode_attention(q, k, k, return_stats=True)[1]["cluster"] == 0


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("batch,skv,splits", [(1, 129, 3), (3, 700, 1), (2, 64, 16)])
def test_a_call_that_names_its_splits_leaves_its_partials(batch, skv, splits, paged):
    """Calls this small run on clusters when the split count is left open. With one, the scratch is the caller's: its
    partials, merged on the host, are the output."""
    import torch
    from scicompute_attention_b200 import _lib, ops
    dt, hq, hkv, d, bs = ol.DT_F16, 8, 2, 128, 16
    gen = torch.Generator("cuda").manual_seed(9)
    q = torch.randn(batch, hq, 1, d, device="cuda", dtype=torch.float16, generator=gen)
    if paged:
        width = -(-skv // bs)
        k, v = (torch.randn(batch * width, bs, hkv, d, device="cuda", dtype=torch.float16, generator=gen) for _ in range(2))
        table = torch.randperm(batch * width, device="cuda", generator=gen).to(torch.int32).view(batch, width)
        lens = torch.full((batch,), skv, device="cuda", dtype=torch.int32)
    else:
        k, v = (torch.randn(batch, hkv, skv, d, device="cuda", dtype=torch.float16, generator=gen) for _ in range(2))
    base = batch * hq * splits
    ws = torch.full((base * (2 + d),), float("nan"), device="cuda")
    out = torch.empty_like(q)
    p = _lib.DecodeFwdParams()
    p.q, p.k, p.v, p.out = q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr()
    p.partial_m, p.partial_l, p.partial_o = (ws.data_ptr() + 4 * base * i for i in range(3))
    p.batch, p.num_heads, p.num_kv_heads, p.seq_kv, p.head_dim, p.num_splits = batch, hq, hkv, skv, d, splits
    p.q_stride = p.o_stride = _lib.DecodeStrides(hq * d, d, d)
    p.k_stride = p.v_stride = _lib.DecodeStrides(0, d, hkv * d) if paged else _lib.DecodeStrides(hkv * skv * d, skv * d, d)
    p.scale, p.dtype = ops.effective_scale(None, d), dt
    if paged:
        p.page_table, p.seq_lens = table.data_ptr(), lens.data_ptr()
        p.block_size, p.max_blocks_per_seq, p.num_kv_blocks = bs, width, batch * width
    lib, stream = _lib.lib(), torch.cuda.current_stream().cuda_stream
    _lib.check((lib.sca_launch_decode_splitk_paged if paged else lib.sca_launch_decode_splitk)(C.byref(p), stream))
    m, l = ws[:base].view(-1, splits).double(), ws[base:2 * base].view(-1, splits).double()
    o = ws[2 * base:].view(-1, splits, d).double()
    used = m > -float("inf")  # the other slots are marked empty
    assert used.any(1).all()
    weight = torch.where(used, torch.exp(m - m.amax(1, keepdim=True)), 0.0)
    o = torch.where(used[..., None], o, 0.0)
    l = torch.where(used, l, 0.0)
    expect = (weight[..., None] * o).sum(1) / (weight * l).sum(1, keepdim=True)
    # one rounding to fp16 (2^-11 relative of the value) behind fp32 sums
    assert torch.allclose(out.view(-1, d).double(), expect, rtol=2 ** -10, atol=2 ** -14)
    # the same call with the split count left open: one launch, the scratch stays as it was
    ws.fill_(float("nan"))
    cluster = C.c_int32(0)
    _lib.check(lib.sca_launch_decode_auto(C.byref(p), C.byref(cluster), stream))
    assert cluster.value > 0 and torch.isnan(ws).all()
    assert torch.allclose(out.view(-1, d).double(), expect, rtol=2 ** -10, atol=2 ** -14)
