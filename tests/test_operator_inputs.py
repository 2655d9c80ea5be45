"""Tensors the operators cannot address - wrong strides, index lists of another type or too short, another type than the pool's -
are refused before anything is launched, by the general form (on the CPU, with the launch layer replaced) and by the native one."""
import numpy as np
import pytest
import torch

from scicompute_attention_b200 import _lib, ops

BF, I32 = torch.bfloat16, torch.int32
B, HQ, HKV, S, D, BS, NB = 2, 4, 2, 24, 64, 16, 6


def _calls(dev):
    """(name, call) pairs; every call takes the keywords of the operator."""
    t = lambda *shape, dtype=BF: torch.zeros(shape, dtype=dtype, device=dev)
    ints = lambda *shape: torch.zeros(shape, dtype=I32, device=dev)
    q, q1, k = t(B, HQ, S, D), t(B, HQ, 1, D), t(B, HKV, S, D)
    pool, new = t(NB, BS, HKV, D), t(3, HKV, D)
    table, lens, slots = ints(B, 4), ints(B), ints(3)
    flat_q, flat_k = t(S, HQ, D), t(S, HKV, D)
    cu, total = np.array([0, S], np.int32), np.array([S], np.int32)
    turned, repeated = t(B, HKV, D, S).transpose(2, 3), t(B, HKV, 1, D).expand(B, HKV, S, D)
    wide_pool, wide_table = t(NB, BS, 2 * HKV, D)[:, :, :HKV], ints(B, 9)[:, :4]
    paged = lambda q_=q1, k_=pool, v_=pool, table_=table, lens_=lens: lambda **w: ops.paged_attention(q_, k_, v_, table_, lens_, block_size=BS, **w)
    chunk = lambda q_=flat_q, k_=pool, v_=pool, table_=ints(1, 4): lambda **w: ops.flash_attention_paged(q_, k_, v_, table_, cu, total, **w)
    append = lambda k_=pool, v_=pool, kn=new, vn=new, slots_=slots: lambda **w: ops.kv_append(k_, v_, kn, vn, slots_, **w)
    batched = lambda k_=pool, v_=pool, kn=new[:B], vn=new[:B], table_=table, lens_=lens: lambda **w: ops.kv_append_batched(k_, v_, kn, vn, table_, lens_, **w)
    return [
        ("flash, v turned", lambda **w: ops.flash_attention(q, k, turned, **w)),
        ("flash, v repeated", lambda **w: ops.flash_attention(q, k, repeated, **w)),
        ("simt, v turned", lambda **w: ops.simt_attention(q.float(), k.float(), turned.float().contiguous().transpose(2, 3).contiguous().transpose(2, 3), **w)),
        ("decode, v repeated", lambda **w: ops.decode_attention(q1, k, repeated, **w)),
        ("decode, long lengths", lambda **w: ops.decode_attention(q1, k, k, seq_lens=lens.long(), **w)),
        ("decode, few lengths", lambda **w: ops.decode_attention(q1, k, k, seq_lens=lens[:1], **w)),
        ("decode, strided lengths", lambda **w: ops.decode_attention(q1, k, k, seq_lens=ints(2 * B)[::2], **w)),
        ("paged, q strided", paged(q_=t(B, 2 * HQ, 1, D)[:, ::2])),
        ("paged, pool sliced", paged(k_=wide_pool, v_=wide_pool)),
        ("paged, v pool sliced", paged(v_=wide_pool)),
        ("paged, table sliced", paged(table_=wide_table)),
        ("paged, pool of another type", paged(k_=pool.half(), v_=pool.half())),
        ("paged, long lengths", paged(lens_=lens.long())),
        ("paged, few lengths", paged(lens_=lens[:1])),
        ("varlen, types", lambda **w: ops.flash_attention_varlen(flat_q, flat_k.half(), flat_k.half(), cu, cu, **w)),
        ("varlen, head dims", lambda **w: ops.flash_attention_varlen(flat_q, t(S, HKV, 128), t(S, HKV, 128), cu, cu, **w)),
        ("chunk, types", chunk(k_=pool.half(), v_=pool.half())),
        ("chunk, table sliced", chunk(table_=ints(2, 9)[:, :4])),
        ("append, few slots", append(slots_=slots[:2])),
        ("append, long slots", append(slots_=slots.long())),
        ("append, strided slots", append(slots_=ints(6)[::2])),
        ("append, strided rows", append(kn=t(3, 2 * HKV, D)[:, ::2])),
        ("append, narrow rows", append(kn=t(3, HKV, D // 2), vn=t(3, HKV, D // 2))),
        ("append, few v rows", append(vn=new[:2])),
        ("append, rows of another type", append(kn=new.half(), vn=new.half())),
        ("append, pool sliced", append(k_=wide_pool, v_=wide_pool)),
        ("append, v pool smaller", append(v_=pool[:3])),
        ("batched, long table", batched(table_=table.long())),
        ("batched, table sliced", batched(table_=wide_table)),
        ("batched, few table rows", batched(table_=table[:1])),
        ("batched, few lengths", batched(lens_=lens[:1])),
        ("batched, narrow rows", batched(kn=t(B, HKV, D // 2), vn=t(B, HKV, D // 2))),
        ("reset, long ids", lambda **w: ops.kv_reset(pool, pool, slots.long(), **w)),
        ("reset, pool sliced", lambda **w: ops.kv_reset(wide_pool, wide_pool, slots, **w)),
        ("gather, long ids", lambda **w: ops.kv_gather(pool, slots.long(), **w)),
        ("gather, strided ids", lambda **w: ops.kv_gather(pool, ints(6)[::2], **w)),
        ("gather, pool sliced", lambda **w: ops.kv_gather(wide_pool, slots, **w)),
    ]


NAMES = [name for name, _ in _calls("meta")]


def _general_only(dev):
    """Arguments and operators that have no native form."""
    t = lambda *shape, dtype=BF: torch.zeros(shape, dtype=dtype, device=dev)
    q, k = t(B, HQ, S, D), t(B, HKV, S, D)
    turned = t(B, HKV, D, S).transpose(2, 3)
    return [lambda: ops.decode_triples(q[:, :, :1].contiguous(), k, turned), lambda: ops.decode_partials(q[:, :, :1].contiguous(), k, turned),
            lambda: ops.decode_triples(q, k, k), lambda: ops.naive_attention(q, k, turned), lambda: ops.merge_triples(t(2, 8, D + 2), BF),
            lambda: ops.flash_attention(q, k, k, out=q[:, :2]), lambda: ops.flash_attention(q, k, k, out=torch.zeros_like(q, dtype=torch.float16)),
            lambda: ops.flash_attention(q, k, k, out=torch.zeros_like(q), lse=t(B, HQ, 3, dtype=torch.float32), return_lse=True)]


class _NoLaunch:
    def __getattr__(self, name):
        raise AssertionError(f"{name} called")


@pytest.fixture
def no_launch(monkeypatch):
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: None)
    monkeypatch.setattr(ops, "lib", _NoLaunch)
    monkeypatch.setattr(ops, "_stream_ptr", lambda stream=None: 0)
    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "acquire_scratch_fp32", lambda n, device, **w: torch.empty(n))


@pytest.mark.parametrize("i", range(len(NAMES)), ids=NAMES)
def test_general_form(no_launch, i):
    with pytest.raises(_lib.ScaError) as e:
        _calls("cpu")[i][1]()
    assert e.value.code == 4


@pytest.mark.parametrize("i", range(8))
def test_forms_without_a_native_one(no_launch, i):
    with pytest.raises(_lib.ScaError) as e:
        _general_only("cpu")[i]()
    assert e.value.code == 4


@pytest.mark.gpu
@pytest.mark.parametrize("i", range(len(NAMES)), ids=NAMES)
def test_native_form(i, monkeypatch):
    call = _calls("cuda")[i][1]
    monkeypatch.setattr(ops, "lib", _NoLaunch)  # the general form has nothing to launch with
    said = []
    for w in ({}, {"stream": torch.cuda.current_stream()}):
        with pytest.raises(_lib.ScaError) as e:
            call(**w)
        said.append((e.value.code, e.value.message))
    assert said[0] == said[1] and said[0][0] == 4


@pytest.mark.gpu
def test_lengths_on_the_host():
    q, k = (torch.zeros((B, h, n, D), dtype=BF, device="cuda") for h, n in ((HQ, 1), (HKV, S)))
    with pytest.raises(_lib.ScaError) as e:
        ops.decode_attention(q, k, k, seq_lens=torch.tensor([S, S], dtype=I32))
    assert e.value.code == 5


@pytest.mark.gpu
def test_forms_that_stay_accepted():
    """Longer index lists, rows in another shape, raw words of the pool's width, a larger V pool, leading rows of larger tensors."""
    g = torch.Generator(device="cuda").manual_seed(2)
    pool = torch.randn((NB, BS, HKV, D), device="cuda", generator=g).to(BF)
    new = torch.randn((3, HKV, D), device="cuda", generator=g).to(BF)
    slots = torch.tensor([5, -1, 40, 7, 8], dtype=I32, device="cuda")
    want = pool.clone()
    want.view(-1, HKV, D)[[5, 40]] = new[[0, 2]]
    for kn in (new, new.view(3, 1, HKV, D), new.view(3, HKV * D), new.view(torch.int16), torch.cat([new, new])[:3]):
        k, v = pool.clone(), torch.cat([pool, pool])
        ops.kv_append(k, v, kn, torch.cat([new, new]), slots)
        assert torch.equal(k, want) and torch.equal(v[:NB], want) and torch.equal(v[NB:], pool)
    table = torch.arange(NB, dtype=I32, device="cuda").view(3, 2)
    lens = torch.tensor([20, 32, 9, 1], dtype=I32, device="cuda")
    q = torch.randn((2, HQ, 1, D), device="cuda", generator=g).to(BF)
    assert torch.equal(ops.paged_attention(q, pool, pool, table, lens, block_size=BS), ops.paged_attention(q, pool, pool, table[:2], lens[:2], block_size=BS))
    k = pool.view(3, BS * 2, HKV, D).permute(0, 2, 1, 3).contiguous()[:2]
    assert torch.equal(ops.decode_attention(q, k, k, seq_lens=lens), ops.decode_attention(q, k, k, seq_lens=lens[:2]))
