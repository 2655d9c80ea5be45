"""The native operators on top of a library whose launches only count themselves and return a chosen status: a launch that failed
is not tried again, its error is raised; a refusal is left to the general form."""
import os
import shutil
import subprocess
import sys
import sysconfig

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LAUNCHES = ("flash_fwd", "simt_forward", "decode_auto", "flash_varlen", "flash_paged", "kv_append", "kv_append_batched", "kv_reset_block", "kv_gather")
STUB = "int status, launches;\nlong long sca_flash_varlen_workspace_bytes(void) { return 4096; }\n" + "".join(
    f"int sca_launch_{name}(void) {{ ++launches; return status; }}\n" for name in LAUNCHES)
SCRIPT = """
import ctypes, importlib.util, sys, types
import numpy as np
import torch
stub = ctypes.CDLL(sys.argv[1])
status, launches = (ctypes.c_int.in_dll(stub, n) for n in ("status", "launches"))
spec = importlib.util.spec_from_file_location("_native", sys.argv[2])
native = importlib.util.module_from_spec(spec)
spec.loader.exec_module(native)
class Failed(Exception): pass
def check(rc): raise Failed(rc)
native.init(types.SimpleNamespace(pool={}), lambda n, device: torch.empty(n, device=device), check)
t = lambda *shape: torch.zeros(shape, device="cuda", dtype=torch.float16)
q, q1, k, pool, rows = t(1, 4, 8, 64), t(1, 4, 1, 64), t(1, 2, 8, 64), t(4, 16, 2, 64), t(1, 2, 64)
table, ids = (torch.zeros(s, device="cuda", dtype=torch.int32) for s in ((1, 4), (1,)))
cu, lens = np.array([0, 8], np.int32), np.array([8], np.int32)
calls = {"flash": (q, k, k, False, None, False, "bhsd", False), "decode": (q1, k, k, None, "bhsd", None),
         "paged": (q1, pool, pool, table, ids, 16, None, 0, 0), "varlen": (t(8, 4, 64), t(8, 2, 64), t(8, 2, 64), cu, cu, True, None),
         "chunk": (t(8, 4, 64), pool, pool, table, cu, lens, True, None), "append": (pool, pool, rows, rows, ids),
         "append_batched": (pool, pool, rows, rows, table, ids), "reset": (pool, pool, ids), "gather": (pool, ids)}
for name, args in [*calls.items(), ("flash", calls["flash"][:7] + (True,))]:
    for rc in (0, 4, 5, 100, 101, 102, 500):
        status.value, launches.value = rc, 0
        try:
            got = getattr(native, name)(*args)
            assert (got is None) == (rc in (4, 5)) and rc < 100, (name, rc, got)
        except Failed as e:
            assert rc >= 100 and e.args == (rc,), (name, rc)
        assert launches.value == 1, (name, rc, launches.value)
print("ok")
"""


def test_one_launch_and_its_error(tmp_path):
    from scicompute_attention_b200 import build
    subprocess.run(["gcc", "-shared", "-fPIC", "-x", "c", "-", "-o", str(tmp_path / "libsca_b200.so")], input=STUB, text=True, check=True)
    module = shutil.copy(build.NATIVE_OPS, tmp_path / ("_native" + sysconfig.get_config_var("EXT_SUFFIX")))
    run = subprocess.run([sys.executable, "-c", SCRIPT, str(tmp_path / "libsca_b200.so"), str(module)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stderr
