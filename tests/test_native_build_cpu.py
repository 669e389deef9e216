"""The CPython extension belongs to one torch and one interpreter: another one's is rebuilt or left alone, and without it the
Python operators take every call."""
import sys

import pytest
import torch

from moespresso_b200 import _abi, _build
from moespresso_b200 import _torchabi as _t
from moespresso_b200.qwen import full_attention as fa


@pytest.mark.parametrize("what", ["torch", "commit", "abi", "python", "flags"])
def test_stamp_follows_what_the_extension_was_built_against(monkeypatch, what):
    _build.build()
    assert _build.is_current()
    if what == "torch":
        monkeypatch.setattr(torch, "__version__", "2.99.0")
    elif what == "commit":
        monkeypatch.setattr(torch.version, "git_version", "0" * 40)
    elif what == "abi":
        monkeypatch.setattr(torch._C, "_GLIBCXX_USE_CXX11_ABI", not torch._C._GLIBCXX_USE_CXX11_ABI)
    elif what == "python":
        monkeypatch.setattr(sys, "version", "3.99.0")
    else:
        monkeypatch.setattr(_build, "GXX_FLAGS", [*_build.GXX_FLAGS, "-DX"])
    assert not _build.native_is_current() and _build.library_is_current()


def _broken_build():
    raise RuntimeError("no compiler")


@pytest.mark.parametrize("how", ["stale and no compiler", "does not load"])
def test_python_operators_without_the_extension(monkeypatch, how):
    monkeypatch.setattr(_t, "_native", None)
    monkeypatch.setitem(sys.modules, "moespresso_b200._native", None)      # an import of it raises ImportError
    if hasattr(sys.modules["moespresso_b200"], "_native"):
        monkeypatch.delattr("moespresso_b200._native")
    if how != "does not load":
        monkeypatch.setattr(_build, "native_is_current", lambda: False)
        monkeypatch.setattr(_build, "build_native", _broken_build)
    x = torch.zeros(1, 2, 1, 256)
    with pytest.warns(RuntimeWarning, match="no native host calls"):
        assert _t.native("q8_decode", x, x, x, x, x, x, x, 0.1, 4) is None
    assert _t._native is False
    launched = []
    monkeypatch.setattr(fa, "require_cuda", lambda *tensors: torch.device("cpu"))
    monkeypatch.setattr(fa, "_q8_pair", lambda *a: launched.append(a[0]))
    cache = fa.QuantizedKVCache(2, 256, 8, device="cpu")
    cache.update_and_fetch(torch.ones(1, 2, 3, 256), torch.ones(1, 2, 3, 256))
    assert launched == ["affine_q8_append"] and cache.offset == 3


def test_a_missing_extension_does_not_keep_the_library_from_loading(monkeypatch):
    monkeypatch.setattr(_abi, "_lib", None)
    monkeypatch.setattr(_build, "NATIVE", _build.NATIVE + ".missing")
    monkeypatch.setattr(_build, "build_native", _broken_build)
    monkeypatch.setattr(_build, "build_library", _broken_build)
    assert _build.library_is_current() and not _build.is_current()
    assert _abi.load().mxb_abi_version() == 1


def test_a_rebuild_leaves_the_loaded_extension_alone():
    """Ranks that start together may each build: the file is replaced whole, what another process has mapped stays."""
    import os
    _build.build()
    before = os.stat(_build.NATIVE).st_ino
    held = open(_build.NATIVE, "rb")
    _build.build_native()
    assert os.stat(_build.NATIVE).st_ino != before and os.fstat(held.fileno()).st_ino == before
    assert held.read(4) == b"\x7fELF" and _build.is_current()
    assert not [n for n in os.listdir(os.path.join(_build.HERE, "build")) if n.endswith(".part")]
    held.close()
