"""Offsets of a packed batch that go up and down between the right ends are refused before anything is sized by them: the entries
they describe are without bound, and an allocation that fails has no place at a C entry."""
import ctypes as C

import numpy as np
import pytest

from scicompute_attention_b200 import _lib

BIG = 2**31 - 1
PAIRS, TOTAL = 300, 128  # 600 sequences, half of them of 2^31 - 1 tokens: 2e10 entries of 32 tokens
BAD = {"up and down": [0] + [BIG, 0] * PAIRS + [TOTAL], "empty": [0, 64, 64, TOTAL], "down": [0, 96, 64, TOTAL], "negative": [0, -5, TOTAL]}


def _addresses():
    """16-byte aligned numbers in the place of tensors: a refused call looks at none of them."""
    return (C.c_void_p(0x10000 * (i + 1)) for i in range(4))


@pytest.mark.parametrize("causal", (0, 1))
@pytest.mark.parametrize("name", BAD)
def test_packed(name, causal):
    cu = np.array(BAD[name], np.int32)
    good = np.linspace(0, TOTAL, len(cu)).astype(np.int32) if name != "up and down" else cu
    for cu_q, cu_kv in ((cu, good), (good, cu)):
        p = _lib.FlashVarlenParams()
        p.q, p.k, p.v, p.out = _addresses()
        p.total_q = p.total_kv = TOTAL
        p.num_heads, p.num_kv_heads, p.head_dim, p.num_seqs, p.scale, p.causal, p.dtype_id = 4, 2, 64, len(cu) - 1, 0.125, causal, _lib.DTYPE_BF16
        p.cu_seqlens_q, p.cu_seqlens_kv = cu_q.ctypes.data, cu_kv.ctypes.data
        with pytest.raises(_lib.ScaError) as e:
            _lib.check(_lib.lib().sca_launch_flash_varlen(C.byref(p), None))
        assert e.value.code == 4 and "sequence" in e.value.message


@pytest.mark.parametrize("name", BAD)
def test_paged(name):
    cu = np.array(BAD[name], np.int32)
    lens = np.full(len(cu) - 1, 200, np.int32)
    p = _lib.FlashPagedParams()
    p.q, p.out, p.k_pool, p.v_pool = _addresses()
    p.page_table = C.c_void_p(0x90000)
    p.total_q, p.num_heads, p.num_kv_heads, p.head_dim, p.num_seqs = TOTAL, 4, 2, 64, len(lens)
    p.num_blocks, p.block_size, p.max_blocks_per_seq, p.scale, p.dtype_id = 64, 16, 16, 0.125, _lib.DTYPE_BF16
    p.cu_seqlens_q, p.seq_lens_kv = cu.ctypes.data, lens.ctypes.data
    with pytest.raises(_lib.ScaError) as e:
        _lib.check(_lib.lib().sca_launch_flash_paged(C.byref(p), None))
    assert e.value.code == 4 and "sequence" in e.value.message


@pytest.mark.gpu
def test_operators():
    import torch
    from scicompute_attention_b200 import ops
    cu = np.array(BAD["up and down"], np.int32)
    q, k = (torch.zeros((TOTAL, h, 64), dtype=torch.bfloat16, device="cuda") for h in (4, 2))
    pool, table = torch.zeros((64, 16, 2, 64), dtype=torch.bfloat16, device="cuda"), torch.zeros((len(cu) - 1, 16), dtype=torch.int32, device="cuda")
    calls = (lambda **w: ops.flash_attention_varlen(q, k, k, cu, cu, **w),
             lambda **w: ops.flash_attention_paged(q, pool, pool, table, cu, np.full(len(cu) - 1, 200, np.int32), **w))
    for call in calls:
        said = []
        for w in ({}, {"stream": torch.cuda.current_stream()}):
            with pytest.raises(_lib.ScaError) as e:
                call(**w)
            said.append((e.value.code, e.value.message))
        assert said[0] == said[1] and said[0][0] == 4
