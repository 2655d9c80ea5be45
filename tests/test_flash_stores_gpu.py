"""The two widths of the prefill's output stores: 32 bytes where every row of the output starts on a 32-byte boundary, 16 bytes
otherwise. Both write the same bits and nothing else."""
import pytest

import oracle_lib as ol
import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", (32, 64, 96, 128, 160, 192, 256))
@pytest.mark.parametrize("dt", (ol.DT_F16, ol.DT_BF16))
def test_output_at_a_16_byte_boundary(dt, d):
    import torch
    from scicompute_attention_b200 import ops
    b, hq, hkv, s = 2, 4, 2, 131
    q, k, v = (H.to_device(H.uniform_inputs((b, h, s, d), 70 + i, dt)[0], dt) for i, h in enumerate((hq, hkv, hkv)))
    wide = ops.flash_attention(q, k, v, causal=True)
    assert wide.data_ptr() % 32 == 0
    buf = torch.full((wide.numel() + 64,), 7.0, dtype=wide.dtype, device="cuda")
    first = 8 if buf.data_ptr() % 32 == 0 else 16  # 16 bytes past a 32-byte boundary
    out = buf[first:first + wide.numel()].view(wide.shape)
    assert out.data_ptr() % 32 == 16
    ops.flash_attention(q, k, v, causal=True, out=out)
    torch.cuda.synchronize()
    assert torch.equal(out, wide)
    assert bool((buf[:first] == 7).all()) and bool((buf[first + wide.numel():] == 7).all())
