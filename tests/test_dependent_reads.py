"""Kernels that are set up while the one ahead of them still writes read global memory with ordinary loads only: the read-only
path wants memory that nobody writes while the kernel lives, and the wait for the predecessor does not hold such loads back."""
import glob
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scicompute_attention_b200", "csrc", "kernels")


@pytest.mark.parametrize("path", [p for p in sorted(glob.glob(os.path.join(KERNELS, "*.cu*"))) if os.path.basename(p) != "naive.cu"], ids=os.path.basename)
def test_no_read_only_loads(path):
    code = re.sub(r"//[^\n]*", "", open(path).read())  # naive.cu launches nothing ahead of its predecessor's end
    assert re.findall(r"__ldg\w*|__restrict__|ld\.global\.nc|__ldlu", code) == []
