import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.dirname(os.path.abspath(__file__)), os.path.join(ROOT, "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


@pytest.fixture(scope="session", autouse=True)
def _built_oracle():
    import oracle_lib
    oracle_lib.oracle()  # builds oracle/liboracle.so on first use
    yield


@pytest.fixture(autouse=True)
def _no_launch_gave_up(request):
    """Every barrier wait of the prefill kernel is bounded; no test may end with one that ran out."""
    yield
    if request.node.get_closest_marker("gpu") is None:
        return
    import torch
    if torch.cuda.is_available() and torch.cuda.is_initialized():
        from scicompute_attention_b200 import ops
        torch.cuda.synchronize()
        assert ops.flash_status() == 0
