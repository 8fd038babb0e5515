"""The native front ends are compiled against one version of torch: under another they are rebuilt, and not loaded."""
import shutil

import pytest
import torch

from hipkittens_b200 import _build, _native


def test_another_torch_means_another_build(native_built, monkeypatch):
    built = _build.shim_path("lib", "_torch_front")
    assert built in native_built and _build.built_for_this_torch(built)
    commands = []
    monkeypatch.setattr(_build, "_run", commands.append)
    assert _build.build_torch_front() == built and not commands
    monkeypatch.setattr(torch, "__version__", torch.__version__ + "1")  # the version in the file is a prefix of it
    assert not _build.built_for_this_torch(built)
    assert _build.build_torch_front() == built and len(commands) == 1
    assert f'-DHK_TORCH_VERSION="{torch.__version__}"' in commands[0]


def test_a_build_for_another_torch_is_not_loaded(native_built, monkeypatch):
    monkeypatch.setattr(_native, "_front_module", None)
    monkeypatch.setattr(torch, "__version__", "1.0")
    with pytest.raises(ImportError, match="another version of torch than 1.0"):
        _native._front()
    monkeypatch.undo()
    assert _native._front() is not None


def test_a_file_without_a_version_is_stale(native_built, tmp_path):
    other = tmp_path / "front.so"
    shutil.copy(_build.LIB_PATH, other)
    assert not _build.built_for_this_torch(str(other))
