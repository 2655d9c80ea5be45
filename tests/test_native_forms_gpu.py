"""What the native operators leave to the general form, calls from several threads, and launches where branches of a capture meet."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype="bfloat16"):
    import torch
    return torch.randn(shape, device="cuda").to(getattr(torch, dtype))


def test_wrapped_tensors_are_not_taken():
    import torch
    from scicompute_attention_b200 import ops
    q, k, v = _rand(1, 4, 20, 64), _rand(1, 2, 50, 64), _rand(1, 2, 50, 64)

    class Named(torch.Tensor):
        pass
    native = lambda *t: ops._native().flash(*t, False, None, False, "bhsd", False)
    plain = native(q, k, v)
    assert torch.equal(plain, ops.flash_attention(q, k, v))
    for t in ((q.as_subclass(Named), k, v), (q, k.as_subclass(Named), v), (q, k, v.as_subclass(Named)), (q.to_sparse(), k, v)):
        assert native(*t) is None
    assert torch.equal(ops.flash_attention(q.as_subclass(Named), k, v).as_subclass(torch.Tensor), plain)
    seen = []

    def look(x):
        seen.append(native(x, k, v))
        return x.float().sum()
    torch.func.vmap(look)(q[None])
    torch.func.grad(look)(q.float())
    torch.func.functionalize(look)(q)
    assert seen == [None] * 3
    with pytest.raises(RuntimeError):  # no data to point at: refused, not read
        torch.func.vmap(lambda x: ops.flash_attention(x, k, v))(torch.stack([q, q]))


def test_threads():
    import torch
    from scicompute_attention_b200 import ops
    q, k, v = _rand(2, 8, 1, 64), _rand(2, 8, 40000, 64), _rand(2, 8, 40000, 64)
    x = _rand(1, 8, 130, 64)

    def work(scale, got):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(30):
                got.append((ops.decode_attention(q, k, v, scale=scale), ops.flash_attention(x, k[:1], v[:1], scale=scale, causal=True)))
            torch.cuda.current_stream().synchronize()
    scales = (0.05, 0.1, 0.2, 0.3)
    torch.cuda.synchronize()
    want = [(ops.decode_attention(q, k, v, scale=s), ops.flash_attention(x, k[:1], v[:1], scale=s, causal=True)) for s in scales]
    torch.cuda.synchronize()
    got = [[] for _ in scales]
    threads = [threading.Thread(target=work, args=a) for a in zip(scales, got)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w, results in zip(want, got):
        assert len(results) == 30
        for r in results:
            assert torch.equal(r[0], w[0]) and torch.equal(r[1], w[1])


def test_branches_of_a_capture():
    """A launch behind a fork and one behind a join, each straight behind launches of this library on both branches."""
    import torch
    from scicompute_attention_b200 import ops
    hq, hkv, s, d, bs = 8, 2, 160, 64, 16
    q, k, v = _rand(1, hq, s, d), _rand(1, hkv, 300, d), _rand(1, hkv, 300, d)
    q1 = _rand(1, hq, 1, d)
    slots = torch.randperm(s * hq // hkv, device="cuda").to(torch.int32)
    ids = torch.randperm(len(slots) // bs, device="cuda").to(torch.int32)
    pools = [torch.zeros((len(slots) // bs, bs, hkv, d), device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    side = torch.cuda.Stream()

    def step():
        main = torch.cuda.current_stream()
        a = ops.flash_attention(q, k, v, causal=True)
        side.wait_stream(main)
        with torch.cuda.stream(side):
            one = ops.decode_attention(q1, a, a)
        rows = a.view(-1, hkv, d)
        ops.kv_append(pools[0], pools[1], rows, rows, slots)
        main.wait_stream(side)
        g = ops.kv_gather(pools[0], ids)                                             # behind the append and the decode
        b = ops.flash_attention(one, g.view(1, hkv, -1, d), g.view(1, hkv, -1, d))
        for t in (a, one):
            t.record_stream(side if t is a else main)
        return a, one, g, b
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(10):
        q.copy_(_rand(1, hq, s, d))
        q1.copy_(_rand(1, hq, 1, d))
        for p in pools:
            p.zero_()
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in captured]
        for a, b in zip(got, step()):
            assert torch.equal(a, b)
        torch.cuda.synchronize()
