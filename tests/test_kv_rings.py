"""The K/V rings of the prefill kernel, one per padded head dim and input type, on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_ring_of_the_kernel(tmp_path):
    exe = str(tmp_path / "kv_rings")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", os.path.join(ROOT, "scicompute_attention_b200", "csrc", "kernels"),
                    os.path.join(ROOT, "tests", "cpp", "kv_rings.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = {tuple(map(int, line.split()[:3])): tuple(map(int, line.split()[3:])) for line in out.splitlines()}
    assert len(rows) == 12 and {d for d, _, _ in rows} == {64, 128, 256} and {c for d, c, _ in rows if d == 256} == {0, 4}
    for (dim, converters, plan), seen in rows.items():
        if plan == 0:
            assert seen == (0, 0), (dim, converters, seen)
    assert sum(rows[128, 2, 1]) > 0 and sum(rows[256, 4, 1]) > 0  # the model sees the mistake where K and V share slots
