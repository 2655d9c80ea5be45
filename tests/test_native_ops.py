"""The native form of the operators against their general Python form: the same slots, the same bits, the same refusals."""
import random

import numpy as np
import pytest
import torch

from scicompute_attention_b200 import _lib, ops


def test_slot_rule_is_the_one_of_the_general_form():
    rng = random.Random(3)
    for _ in range(3000):
        args = rng.randint(-1, 5000), rng.randint(0, 3000), rng.randint(1, 400), rng.choice([148, 132, 1])
        assert ops._native().slots(*args) == ops.slots_for_schedule(*args), args


def test_host_tensors_are_left_to_the_general_form():
    t = torch.ones(1, 2, 3, 32, dtype=torch.float16)
    n = ops._native()
    assert n.flash(t, t, t, False, None, False, "bhsd", False) is None
    assert n.decode(t, t, t, None, "bhsd", None) is None
    assert n.gather(t, t) is None and n.flash(1, 2, 3) is None
    with pytest.raises(_lib.ScaError):
        ops.flash_attention(t, t, t)


def _rand(*shape, dtype=torch.bfloat16):
    return torch.randn(shape, device="cuda", dtype=torch.float32).to(dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ("bhsd", "bshd"))
@pytest.mark.parametrize("lse", (False, True))
def test_dense_forms_agree(layout, lse):
    def make(h, s, dtype):
        return _rand(*((2, h, s, 64) if layout == "bhsd" else (2, s, h, 64)), dtype=dtype)
    s = torch.cuda.current_stream()
    for op, dtype in ((ops.flash_attention, torch.bfloat16), (ops.flash_attention, torch.float16), (ops.simt_attention, torch.float32)):
        q, k, v = make(6, 75, dtype), make(3, 90, dtype), make(3, 90, dtype)
        for scale in (None, 0.3, 0.0):
            native = op(q, k, v, causal=True, scale=scale, return_lse=lse, layout=layout)
            general = op(q, k, v, causal=True, scale=scale, return_lse=lse, layout=layout, stream=s)
            for a, b in zip(native, general) if lse else ((native, general),):
                assert a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b)
    q = make(6, 1, torch.bfloat16)
    k, v = make(3, 700, torch.bfloat16), make(3, 700, torch.bfloat16)
    lens = torch.tensor([700, 33], dtype=torch.int32, device="cuda")
    for seq_lens in (None, lens):
        assert torch.equal(ops.decode_attention(q, k, v, layout=layout, seq_lens=seq_lens),
                           ops.decode_attention(q, k, v, layout=layout, seq_lens=seq_lens, stream=s))


@pytest.mark.gpu
def test_paged_and_packed_forms_agree():
    s = torch.cuda.current_stream()
    bs, hq, hkv, d, lens = 16, 8, 2, 128, (500, 17, 260)
    blocks = [-(-n // bs) for n in lens]
    table = torch.full((3, max(blocks)), -1, dtype=torch.int32)
    at = 0
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    table = table.cuda()
    k, v = _rand(at, bs, hkv, d), _rand(at, bs, hkv, d)
    dev_lens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = _rand(3, hq, 1, d)
    for hints in ({}, {"typical_len": 259, "longest_len": 500}):
        assert torch.equal(ops.paged_attention(q, k, v, table, dev_lens, block_size=bs, **hints),
                           ops.paged_attention(q, k, v, table, dev_lens, block_size=bs, stream=s, **hints))
    kn, vn = _rand(3, hkv, d), _rand(3, hkv, d)
    pools = [(k.clone(), v.clone()) for _ in range(2)]
    for (kp, vp), stream in zip(pools, (None, s)):
        ops.kv_append_batched(kp, vp, kn, vn, table, dev_lens, stream=stream)
        ops.kv_append(kp, vp, kn, vn, torch.tensor([5, 90, 333], dtype=torch.int32, device="cuda"), stream=stream)
        ops.kv_reset(kp, vp, torch.tensor([2, 7], dtype=torch.int32, device="cuda"), stream=stream)
    assert torch.equal(pools[0][0], pools[1][0]) and torch.equal(pools[0][1], pools[1][1])
    ids = torch.tensor([9, 0, 4], dtype=torch.int32, device="cuda")
    assert torch.equal(ops.kv_gather(k, ids), ops.kv_gather(k, ids, stream=s))
    new = (40, 17, 3)
    cu = np.concatenate([[0], np.cumsum(new)]).astype(np.int32)
    qp = _rand(sum(new), hq, d)
    host_lens = np.array(lens, np.int32)
    assert torch.equal(ops.flash_attention_paged(qp, k, v, table, cu, host_lens), ops.flash_attention_paged(qp, k, v, table, cu, host_lens, stream=s))
    kp, vp = _rand(sum(new), hkv, d), _rand(sum(new), hkv, d)
    native = ops.flash_attention_varlen(qp, kp, vp, cu, cu, causal=True)
    assert torch.equal(native, ops.flash_attention_varlen(qp, kp, vp, cu, cu, causal=True, stream=s))
    assert torch.equal(native, ops.flash_attention_varlen(qp, kp, vp, cu.tolist(), cu.astype(np.int64), causal=True))  # other host forms


@pytest.mark.gpu
def test_refusals_are_those_of_the_general_form():
    q, k = _rand(1, 4, 8, 64), _rand(1, 2, 8, 64)
    calls = [lambda **w: ops.flash_attention(q, k, k[:, :, :4], **w), lambda **w: ops.flash_attention(q, k[..., ::2], k[..., ::2], **w),
             lambda **w: ops.flash_attention(q, k, k, layout="shbd", **w), lambda **w: ops.flash_attention(q, k[:, :, :4].contiguous(), k[:, :, :4].contiguous(), causal=True, **w),
             lambda **w: ops.flash_attention(q.float(), k.float(), k.float(), **w), lambda **w: ops.flash_attention(q[..., :40].contiguous(), k[..., :40].contiguous(), k[..., :40].contiguous(), **w),
             lambda **w: ops.decode_attention(q, k, k, **w), lambda **w: ops.decode_attention(q[:, :3, :1].contiguous(), k, k, **w),
             lambda **w: ops.flash_attention(q, k, k.cpu(), **w), lambda **w: ops.kv_gather(k, torch.tensor([1, 2]), **w)]
    for i, call in enumerate(calls):
        said = []
        for w in ({}, {"stream": torch.cuda.current_stream()}):
            with pytest.raises(_lib.ScaError) as e:
                call(**w)
            said.append((e.value.code, e.value.message))
        assert said[0] == said[1], i


@pytest.mark.gpu
def test_scratch_under_capture_belongs_to_the_graph():
    """A decode call whose partials need scratch: capture takes none of this thread's pool."""
    q, k = _rand(2, 8, 1, 64), _rand(2, 8, 40000, 64)
    eager = ops.decode_attention(q, k, k)
    before = dict(ops._scratch.pool)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = ops.decode_attention(q, k, k)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, eager)
    assert ops._scratch.pool.keys() == before.keys()
