"""How many CTAs share an item, read from the launches themselves: the problems of test_flash_split_gpu.py do run on clusters of
8, 4 and 2, and a problem with an item for every SM, or of few KV tiles, on none."""
import json

import pytest

pytestmark = pytest.mark.gpu

# b, hq, hkv, sq, skv, items: query tiles of 128 rows, the heads of a kv head sharing one where that leaves fewer; then the CTAs
# that share an item: the largest of 8, 4, 2 for which items * CTAs do not exceed 148 SMs, where that saves 4 (D=64), 3 (128) or
# 6 (256) of the steps of 128 keys
CASES = ((1, 2, 1, 100, 1024, 2, 8), (1, 4, 4, 1, 1100, 4, 8), (5, 8, 2, 40, 1701, 20, 4), (10, 4, 4, 128, 1029, 40, {64: 2, 128: 2, 256: 1}),
         (10, 4, 4, 128, 1541, 40, 2), (20, 8, 8, 128, 1029, 160, 1), (1, 4, 4, 100, 256, 4, 1))


def _launches(call, path):
    import torch
    call()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(path))
    kernels = [e for e in json.load(open(path))["traceEvents"] if e.get("cat") == "kernel"]
    if not kernels:
        pytest.skip("launches cannot be traced here")
    kernels = [e for e in kernels if "flash_fwd_sm100_kernel" in e["name"]]
    return [(e["args"]["grid"][0], "true>" in e["name"].replace(" ", "").split("(")[0][-6:]) for e in kernels]


@pytest.mark.parametrize("d", (64, 128, 256))
def test_ctas_per_item(d, tmp_path):
    import numpy as np
    import torch
    from scicompute_attention_b200 import ops
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the cases are for 148 SMs")
    for n, (b, hq, hkv, sq, skv, items, ctas) in enumerate(CASES):
        q, k = (torch.zeros((b, h, s, d), device="cuda", dtype=torch.bfloat16) for h, s in ((hq, sq), (hkv, skv)))
        ctas = ctas[d] if isinstance(ctas, dict) else ctas
        grid = min(items, 148) if ctas == 1 else items * ctas
        assert _launches(lambda: ops.flash_attention(q, k, k, causal=True), tmp_path / f"{n}.json") == [(grid, ctas > 1)], (d, n)
    # one sequence of the same sizes, packed and paged: 2 items of 64 tokens
    q, k = (torch.zeros((s, h, d), device="cuda", dtype=torch.bfloat16) for h, s in ((2, 100), (1, 1024)))
    cu_q, cu_kv = (np.array([0, s], np.int32) for s in (100, 1024))
    pool, table = k.view(64, 16, 1, d), torch.arange(64, device="cuda", dtype=torch.int32).view(1, 64)
    assert _launches(lambda: ops.flash_attention_varlen(q, k, k, cu_q, cu_kv, causal=True), tmp_path / "v.json") == [(16, True)]
    assert _launches(lambda: ops.flash_attention_paged(q, pool, pool, table, cu_q, cu_kv[1:]), tmp_path / "p.json") == [(16, True)]
