"""Calls whose lists lie in host memory, captured into a graph: the replays find them after the caller's arrays, and everything the
call allocated, are gone."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _junk():
    return [np.full(n, -7, np.int32) for n in (8, 16, 32, 64, 128, 256, 1024, 4096) for _ in range(50)]  # takes freed memory over


def test_packed_and_paged_prefill():
    import torch
    from scicompute_attention_b200 import ops
    hq, hkv, d, bs = 8, 2, 64, 16
    lens, new = (300, 17, 900), (40, 17, 200)
    cu, cu_new = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (lens, new))
    rand = lambda *s: torch.randn(s, device="cuda").to(torch.bfloat16)
    q, k, v, qn = rand(cu[-1], hq, d), rand(cu[-1], hkv, d), rand(cu[-1], hkv, d), rand(cu_new[-1], hq, d)
    blocks = [-(-n // bs) for n in lens]
    table = torch.full((3, max(blocks)), -1, dtype=torch.int32)
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(sum(blocks[:i]), sum(blocks[:i + 1]))
    table = table.cuda()
    pool = rand(sum(blocks), bs, hkv, d)
    host_lens = np.array(lens, np.int32)

    def step(c, cn, hl):
        return ops.flash_attention_varlen(q, k, v, c, c, causal=True), ops.flash_attention_paged(qn, pool, pool, table, cn, hl)
    step(cu, cu_new, host_lens)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    mine = [a.copy() for a in (cu, cu_new, host_lens)]
    with torch.cuda.graph(graph):
        captured = step(*mine)
    for a in mine:
        a[:] = -1
    del mine
    kept = _junk()
    for _ in range(5):
        q.copy_(rand(*q.shape))
        qn.copy_(rand(*qn.shape))
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in captured]
        for a, b in zip(got, step(cu, cu_new, host_lens)):
            assert torch.equal(a, b)
        torch.cuda.synchronize()
    assert kept


def test_block_ids_on_the_host():
    import torch
    from scicompute_attention_b200 import _lib
    pool = torch.randn((40, 16, 2, 64), device="cuda").to(torch.bfloat16)
    want = np.array([7, 0, 39, 12], np.int32)
    out = torch.zeros((4, 16, 2, 64), device="cuda", dtype=torch.bfloat16)
    shape = _lib.KvCacheShape(40, 16, 2, 64)
    gather = lambda ids: _lib.check(_lib.lib().sca_launch_kv_gather(pool.data_ptr(), ids.ctypes.data, 4, out.data_ptr(), C.byref(shape), 2,
                                                                    torch.cuda.current_stream().cuda_stream))
    gather(want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    ids = want.copy()
    with torch.cuda.graph(graph):
        gather(ids)
    ids[:] = 3
    del ids
    kept = _junk()
    for _ in range(3):
        pool.copy_(torch.randn(pool.shape, device="cuda"))
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, pool[torch.from_numpy(want).long().cuda()])
    assert kept
