"""Query heads that share a tile, and the moving reference point of the softmax, against the FP64 oracle."""
import numpy as np
import pytest

import helpers as H
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,batch,hq,hkv,sq,skv,d,causal,layout", [
    (ol.DT_BF16, 1, 8, 2, 1, 700, 128, True, "bhsd"),      # four rows of a tile
    (ol.DT_F16, 2, 8, 2, 32, 33, 64, True, "bshd"),        # exactly one packed tile, one key past the diagonal
    (ol.DT_BF16, 1, 32, 8, 65, 129, 128, True, "bshd"),    # one token into the third tile of a head group
    (ol.DT_F16, 1, 6, 3, 190, 190, 128, True, "bhsd"),     # pairs
    (ol.DT_BF16, 1, 6, 2, 130, 257, 128, False, "bhsd"),   # a group of three: heads stay alone
    (ol.DT_F16, 1, 16, 2, 40, 100, 256, True, "bhsd"),     # eight heads in two packs of four
    (ol.DT_BF16, 1, 64, 8, 600, 600, 64, True, "bhsd"),    # more tiles than SMs: two per item
    (ol.DT_BF16, 2, 8, 2, 257, 300, 128, False, "bhsd"),   # a row into the third tile, no mask: shared
    (ol.DT_F16, 2, 8, 2, 384, 400, 128, False, "bshd"),    # whole tiles, no mask: every head alone
    (ol.DT_BF16, 17, 8, 4, 256, 300, 64, True, "bhsd"),    # 68 kv heads and whole tiles: every head alone
])
def test_packed_heads_match_the_oracle(dt, batch, hq, hkv, sq, skv, d, causal, layout):
    from scicompute_attention_b200 import ops
    qb, qd = H.normal_inputs((batch, hq, sq, d), 76000, dt)
    kb, kd = H.normal_inputs((batch, hkv, skv, d), 76001, dt)
    vb, vd = H.uniform_inputs((batch, hkv, skv, d), 76002, dt)
    swap = (lambda x: x) if layout == "bhsd" else (lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3)))
    out, lse = ops.flash_attention(*[H.to_device(swap(x), dt) for x in (qb, kb, vb)], causal=causal, return_lse=True, layout=layout)
    expect, elog = ol.attention_f64(qd, kd, vd, causal=causal, want_lse=True)
    H.check_close(H.to_host_f32(out), expect, dt)
    assert np.abs(lse.cpu().numpy() - elog).max() <= 1e-3


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("shape", ["ramp", "spike"])
def test_scores_that_keep_growing(d, shape):
    """Every KV tile (ramp) or single late keys of it (spike) exceed the running reference point of the softmax."""
    from scicompute_attention_b200 import ops
    dt, sk = ol.DT_F16, 500
    pos = np.arange(sk, dtype=np.float32)[None, None, :, None]
    grow = pos / 40 + 0.1 if shape == "ramp" else 1 + 10 * ((pos % 128) == 100) * (pos / 200)
    q = H.normal_inputs((1, 4, 300, d), 77000, dt)[1]
    kb, kd = ol.encode((H.normal_inputs((1, 2, sk, d), 77001, dt)[1] * grow).astype(np.float32), dt)
    vb, vd = H.uniform_inputs((1, 2, sk, d), 77002, dt)
    qb, qd = ol.encode(q, dt)
    out = ops.flash_attention(*[H.to_device(x, dt) for x in (qb, kb, vb)], causal=True)
    H.check_close(H.to_host_f32(out), ol.attention_f64(qd, kd, vd, causal=True), dt)


def test_a_work_list_sized_for_unpacked_heads_is_still_accepted():
    """A caller that sized the scratch area for one entry per 128 query rows gets fewer heads per tile, not an error."""
    import ctypes as C
    import torch
    from scicompute_attention_b200 import _lib, ops
    lens = [300, 17, 129]
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    q, k, v = (torch.randn(int(cu[-1]), h, 128, device="cuda", dtype=torch.float16, generator=torch.Generator("cuda").manual_seed(i))
               for i, h in enumerate((8, 2, 2)))
    expect = ops.flash_attention_varlen(q, k, v, cu, cu, causal=True)
    out = torch.empty_like(q)
    ws = torch.empty(3 * 16 + (int(cu[-1]) // 128 + 3) * 8, dtype=torch.uint8, device="cuda")
    p = _lib.FlashVarlenParams()
    p.q, p.k, p.v, p.out = q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr()
    p.total_q, p.total_kv, p.num_heads, p.num_kv_heads, p.head_dim, p.num_seqs = int(cu[-1]), int(cu[-1]), 8, 2, 128, 3
    p.cu_seqlens_q = p.cu_seqlens_kv = cu.ctypes.data
    p.scale, p.causal, p.dtype_id = ops.effective_scale(None, 128), 1, ol.DT_F16
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    _lib.check(_lib.lib().sca_launch_flash_varlen(C.byref(p), torch.cuda.current_stream().cuda_stream))
    # the same rows in other tiles: only the order of a row's running sum may differ, 2^-11 relative in fp16
    assert torch.allclose(out.float(), expect.float(), rtol=2e-3, atol=2e-3)
