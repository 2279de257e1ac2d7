"""The autograd node's binary belongs to one torch, and one that cannot be brought up to date is refused."""
import os
import sys

import pytest
import torch

from sp_aurora_b200 import _lib, build, native


def test_the_node_s_file_belongs_to_the_running_torch(monkeypatch):
    path = build.native_path()
    assert native._native.__file__ == str(path) and not build._stale(path, build.NATIVE_DEPS)
    monkeypatch.setattr(torch, "__version__", "99.0")
    assert build.native_path() != path and build._stale(build.native_path(), build.NATIVE_DEPS)


@pytest.mark.parametrize("lib_path", [None, "elsewhere.so"])     # another build of the CUDA library in use
def test_a_failed_rebuild_is_refused_with_the_compiler_s_words(monkeypatch, tmp_path, lib_path):
    old = tmp_path / "node.so"
    old.write_bytes(b"")
    os.utime(old, (1, 1))
    monkeypatch.setattr(build, "native_path", lambda: old)

    def fails(verbose):
        raise RuntimeError("g++ failed: no such member")
    monkeypatch.setattr(build, "_build_native", fails)
    if lib_path:
        monkeypatch.setenv("SPA_LIB_PATH", lib_path)
    failure = _lib._rebuild_if_stale()
    with pytest.raises(ImportError, match="older than its sources(.|\n)*no such member"):
        native._load(failure)
    old.unlink()
    with pytest.raises(ImportError, match="missing(.|\n)*no such member"):
        native._load(failure)


def test_a_missing_compiler_is_a_build_error_that_leaves_a_built_node_usable(monkeypatch, tmp_path):
    path = build.native_path()
    which = build.shutil.which
    monkeypatch.setattr(build.shutil, "which", lambda name: None if name == "g++" else which(name))
    missing = tmp_path / "node.so"
    with monkeypatch.context() as m:
        m.setattr(build, "native_path", lambda: missing)
        failure = _lib._rebuild_if_stale()
    assert isinstance(failure, build.CannotBuild) and "g++ not found" in str(failure)
    monkeypatch.setattr(build, "_stale", lambda *a: True)
    name = native._load(failure).__file__
    assert name == str(path) and sys.modules["sp_aurora_b200.native"] is native
