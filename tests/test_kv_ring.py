"""The K/V ring of the prefill kernel, run on the CPU with loads that land in any order and roles of any speed."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_role_reads_a_tile_that_is_not_there(tmp_path):
    exe = str(tmp_path / "kv_ring_model")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", os.path.join(ROOT, "scicompute_attention_b200", "csrc", "kernels"),
                    os.path.join(ROOT, "tests", "cpp", "kv_ring_model.cpp"), "-o", exe], check=True)
    rows = [tuple(map(int, line.split())) for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert len(rows) == 14
    for plan, slots, converters, early, stuck in rows:
        if plan == 0:  # the kernel's
            assert (early, stuck) == (0, 0), (slots, converters, early, stuck)
        elif slots == 5:  # the model sees both mistakes where K and V share slots
            assert (early if plan == 1 else stuck) > 0, (plan, converters, early, stuck)
