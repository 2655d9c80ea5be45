"""Decode calls small enough for the one-launch cluster kernel, at the edges of its range, against the FP64 oracle."""
import numpy as np
import pytest

import helpers as H
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,batch,hq,hkv,skv,d", [
    (ol.DT_BF16, 1, 8, 8, 1, 128),       # one key: seven CTAs of every cluster hold nothing
    (ol.DT_F16, 1, 4, 1, 449, 64),       # 8 steps for 8 CTAs, the last one with a single key
    (ol.DT_BF16, 1, 32, 8, 1000, 128),   # clusters of 8
    (ol.DT_BF16, 6, 32, 8, 900, 128),    # of 4
    (ol.DT_F16, 16, 32, 8, 500, 128),    # of 2
    (ol.DT_BF16, 2, 32, 1, 700, 128),    # two head chunks of 16 query heads
    (ol.DT_F16, 1, 12, 1, 130, 96),      # 12 heads: both row halves, one of them ragged
    (ol.DT_BF16, 2, 8, 8, 300, 256),     # one CTA per SM
])
def test_cluster_decode_matches_the_oracle(dt, batch, hq, hkv, skv, d):
    import torch
    from scicompute_attention_b200 import ops
    qb, qd = H.normal_inputs((batch, hq, 1, d), 74000, dt)
    kb, kd = H.normal_inputs((batch, hkv, skv, d), 74001, dt)
    vb, vd = H.uniform_inputs((batch, hkv, skv, d), 74002, dt)
    q, k, v = H.to_device(qb, dt), H.to_device(kb, dt), H.to_device(vb, dt)
    H.check_close(H.to_host_f32(ops.decode_attention(q, k, v)), ol.attention_f64(qd, kd, vd, causal=True), dt)
    # ragged, an empty sequence among them: its rows are zero
    lens = np.array([(skv * (i + 1)) // batch for i in range(batch)], dtype=np.int32)
    lens[-1] = 0
    out = H.to_host_f32(ops.decode_attention(q, k, v, seq_lens=torch.from_numpy(lens).cuda()))
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
    out = ops.paged_attention(H.to_device(qb, dt), H.to_device(kb, dt), H.to_device(vb, dt), torch.from_numpy(table).cuda(),
                              torch.from_numpy(lens).cuda(), block_size=block_size)
    expect = ol.paged_decode_f64(qd[:, :, 0], kd, vd, table, lens, block_size)
    H.check_close(H.to_host_f32(out), expect.reshape(seqs, hq, 1, d), dt)
