"""The tiled fp32 kernel at the edges of its tiles, against the FP64 oracle.

Bound: a score is a sum of D products and an output a sum of S_kv terms, accumulated in fp32 (2^-24 relative per
operation, errors of random sign), and ex2.approx adds 2^-22 per weight: below 4e-6 relative L2 with a wide margin for
D <= 256 and S_kv <= 300 (the 128-key case measures 3e-7)."""
import numpy as np
import pytest

import helpers as H
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,hq,hkv,sq,skv,causal,layout", [
    (128, 4, 2, 1, 1, False, "bhsd"),       # one row, one key: the second key group has nothing to do
    (128, 4, 4, 63, 64, True, "bhsd"),
    (128, 4, 1, 65, 129, True, "bshd"),     # one row past the tile, one key past both groups' tiles
    (128, 160, 8, 33, 33, True, "bhsd"),    # more than one wave: the 64-row tile
    (64, 6, 3, 100, 257, False, "bshd"),
    (32, 2, 2, 31, 300, True, "bhsd"),
    (256, 2, 1, 40, 97, True, "bhsd"),      # 32-key tiles
    (160, 2, 2, 64, 33, False, "bhsd"),
    (224, 2, 1, 17, 65, True, "bshd"),
    (256, 256, 64, 17, 17, True, "bhsd"),   # tiles that would be mostly padding: one warp per row
])
def test_tiled_fp32_matches_the_oracle(d, hq, hkv, sq, skv, causal, layout):
    from scicompute_attention_b200 import ops
    dt = ol.DT_F32
    swap = (lambda x: x) if layout == "bhsd" else (lambda x: np.ascontiguousarray(x.transpose(0, 2, 1, 3)))
    arrays = [H.normal_inputs((2, h, n, d), 71000 + i, dt)[1] for i, (h, n) in enumerate(((hq, sq), (hkv, skv), (hkv, skv)))]
    expect, elog = ol.attention_f64(*arrays, causal=causal, want_lse=True)
    out, lse = ops.simt_attention(*[H.to_device(swap(x), dt) for x in arrays], causal=causal, return_lse=True, layout=layout)
    got = H.to_host_f32(out).astype(np.float64)
    rel = np.sqrt(((got - expect) ** 2).sum() / (expect ** 2).sum())
    assert rel <= 4e-6, rel
    assert np.abs(lse.cpu().numpy() - elog).max() <= 1e-5


def test_values_behind_the_causal_mask_do_not_reach_a_row():
    """An infinity or a NaN in a key or value that a row does not see leaves the row alone; the row that sees it shows it."""
    import torch
    from scicompute_attention_b200 import ops
    q, k, v = (torch.randn(1, 2, 70, 64, device="cuda", generator=torch.Generator("cuda").manual_seed(5)) for _ in range(3))
    clean = ops.simt_attention(q, k, v, causal=True)
    v[:, :, 50] = float("inf")
    k[:, :, 60] = float("nan")
    out = ops.simt_attention(q, k, v, causal=True)
    assert torch.equal(out[:, :, :50], clean[:, :, :50])
    assert torch.isinf(out[:, :, 50:60]).all() and torch.isnan(out[:, :, 60:]).all()


def test_rows_that_are_not_16_byte_aligned_still_run():
    import torch
    from scicompute_attention_b200 import ops
    q = torch.randn(2 * 2 * 40 * 64 + 1, device="cuda")[1:].view(2, 2, 40, 64)
    expect = ops.simt_attention(q.clone(), q.clone(), q.clone(), causal=True)
    assert torch.allclose(ops.simt_attention(q, q, q, causal=True), expect, rtol=1e-5, atol=1e-5)
