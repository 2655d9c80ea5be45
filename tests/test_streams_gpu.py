"""Operators launched on a stream that is not the current one, and on two streams at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rand(shape, seed):
    import torch
    return torch.randn(shape, device="cuda", dtype=torch.bfloat16, generator=torch.Generator("cuda").manual_seed(seed))


@pytest.mark.parametrize("paged", [False, True])
def test_the_work_list_lives_until_the_launch_on_its_stream_has_read_it(paged):
    """The stream is held up; meanwhile the current stream takes and fills all memory of the list's size that is free."""
    import torch
    from scicompute_attention_b200 import ops
    lens = np.array([300, 17, 1029, 64], np.int32)
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    q = _rand((int(cu[-1]), 8, 128), 1)
    if paged:
        k, v = _rand((320, 16, 2, 128), 2), _rand((320, 16, 2, 128), 3)
        table = torch.arange(320, dtype=torch.int32, device="cuda").view(4, 80)
        call = lambda stream: ops.flash_attention_paged(q, k, v, table, cu, lens + 100, stream=stream)
    else:
        k, v = _rand((int(cu[-1]), 2, 128), 2), _rand((int(cu[-1]), 2, 128), 3)
        call = lambda stream: ops.flash_attention_varlen(q, k, v, cu, cu, causal=True, stream=stream)
    expect = call(None)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)  # about 10 ms
    out = call(side)
    held = [torch.full((n,), 0x7f, dtype=torch.uint8, device="cuda") for n in (512, 1024, 2048) for _ in range(64)]
    side.synchronize()
    assert torch.equal(out, expect) and ops.flash_status() == 0
    del held


def test_a_result_that_the_current_stream_still_reads_is_not_reused():
    import torch
    from scicompute_attention_b200 import ops
    sets = [[_rand((1, h, 500, 128), 40 + 3 * i + j) for j, h in enumerate((8, 2, 2))] for i in range(2)]
    expect = ops.flash_attention(*sets[0], causal=True)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    out = ops.flash_attention(*sets[0], causal=True, stream=side)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda._sleep(20_000_000)  # about 10 ms
    kept = out.clone()
    del out  # before the copy has run
    for _ in range(4):
        ops.flash_attention(*sets[1], causal=True, stream=side)
    torch.cuda.synchronize()
    assert torch.equal(kept, expect)


def test_decode_on_two_streams_at_once_and_in_threads():
    import threading
    import torch
    from scicompute_attention_b200 import ops
    sets = [[_rand((4, 32, 1, 128), 10 + i), _rand((4, 8, 6000, 128), 20 + i), _rand((4, 8, 6000, 128), 30 + i)] for i in range(2)]
    run = lambda i, stream=None: ops.decode_attention(*sets[i], num_splits=16, stream=stream)
    expect = [run(i) for i in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    a, b = (ops.acquire_scratch_fp32(1000, sets[0][0].device, stream=s) for s in streams)
    assert a.data_ptr() != b.data_ptr()
    for _ in range(20):
        outs = [(i % 2, run(i % 2, streams[i % 2])) for i in range(6)]
        torch.cuda.synchronize()
        assert all(torch.equal(o, expect[i]) for i, o in outs)
    # two threads that launch on the same stream
    wrong = []

    def work(i):
        for _ in range(50):
            out = run(i, streams[0])
            streams[0].synchronize()
            if not torch.equal(out, expect[i]):
                wrong.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_a_captured_decode_does_not_use_the_pool():
    import torch
    from scicompute_attention_b200 import ops
    q, k, v = _rand((4, 32, 1, 128), 1), _rand((4, 8, 6000, 128), 2), _rand((4, 8, 6000, 128), 3)
    expect = ops.decode_attention(q, k, v, num_splits=16)
    graph = torch.cuda.CUDAGraph()
    before = dict(ops._scratch.pool)
    with torch.cuda.graph(graph):
        out = ops.decode_attention(q, k, v, num_splits=16)
    assert ops._scratch.pool.keys() == before.keys()
    for _ in range(3):
        out.zero_()
        graph.replay()
        other = ops.decode_attention(q, k, v, num_splits=16)
        torch.cuda.synchronize()
        assert torch.equal(out, expect) and torch.equal(other, expect)
