"""Which native module the operators take: the one built for this torch and this Python; without it the general form serves."""
import os
import sys
import sysconfig
import types
import warnings

import pytest

import scicompute_attention_b200 as pkg
from scicompute_attention_b200 import build, ops


def test_the_module_in_the_tree_fits():
    assert os.path.basename(build.NATIVE_OPS) == "_native" + sysconfig.get_config_var("EXT_SUFFIX") and os.path.exists(build.NATIVE_OPS)
    assert not os.path.exists(os.path.join(build.PKG, "_native.so"))  # a name that any Python imports
    n = ops._native()
    assert n.__file__ == build.NATIVE_OPS and n.built_with == ops.torch_build()


def _taken(monkeypatch, module):
    monkeypatch.setattr(ops, "_native_module", None)
    monkeypatch.setitem(sys.modules, "scicompute_attention_b200._native", module)
    if module is None:
        monkeypatch.delattr(pkg, "_native", raising=False)
    else:
        monkeypatch.setattr(pkg, "_native", module, raising=False)
    with pytest.warns(RuntimeWarning, match="scicompute_attention_b200.build"):
        n = ops._native()
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert ops._native() is n  # said once
    return n


@pytest.mark.parametrize("module", (None, types.SimpleNamespace(built_with="2.0.0 abc", init=None, flash=None)), ids=("missing", "another torch"))
def test_without_one_the_general_form_serves(monkeypatch, module):
    n = _taken(monkeypatch, module)
    assert n.flash(1, 2, 3) is None and n.append() is None
