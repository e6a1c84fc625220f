"""The call path on torch tensors is tied to what it was built for, and nothing else depends on it."""
import os
import subprocess
import sys

import pytest
import torch

from flash_attn_b200 import _lib, build


def test_a_module_built_for_another_torch_is_built_again_and_not_called(monkeypatch):
    build.build_call()
    assert not build.needs_build_call()
    _lib.load_call()
    monkeypatch.setattr(torch, "__version__", "1.0")
    assert build.needs_build_call()
    with pytest.raises(ImportError, match="flash_attn_b200.build"):
        _lib.load_call()


def test_the_compilers_arguments_count(monkeypatch):
    monkeypatch.setenv("CXX", "another-compiler")
    assert build.needs_build_call()


def test_the_module_carries_the_interpreters_tag():
    import sysconfig
    assert os.path.basename(build.CALL) == "_call" + sysconfig.get_config_var("EXT_SUFFIX")


def test_the_c_entry_points_need_no_call_path():
    code = """
import sys
sys.modules["flash_attn_b200._call"] = None  # (an import of it fails)
from flash_attn_b200 import _lib, num_splits_heuristic
assert _lib.strerror(0) == "success" and num_splits_heuristic(8, 148, 64, 64, 8192) > 1
try:
    _lib.load_call()
except ImportError as e:
    assert "flash_attn_b200.build" in str(e)
else:
    raise AssertionError
"""
    subprocess.check_call([sys.executable, "-c", code], cwd=os.path.dirname(build.PKG))


def test_the_library_is_built_before_the_call_path(monkeypatch):
    order = []
    monkeypatch.setattr(build, "_compile", lambda *a: order.append("library"))
    monkeypatch.setattr(build, "build_call", lambda force=False: order.append("call"))
    build.build(force=True)
    assert order == ["library", "call"]
