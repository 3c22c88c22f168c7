"""The host extension (csrc/host.cpp) is an addition to the library: without it, or with one that is not this torch's, every call takes its general path."""
import importlib.machinery
import importlib.util
import shutil
import subprocess
import sys

import pytest
import torch

from conftest import ROOT

PKG = "sm120-fp4_b200"


def run_without_extension(tmp_path, code):
    """`code` in a copy of the package that holds the library and no extension."""
    shutil.copytree(ROOT / PKG, tmp_path / PKG, ignore=shutil.ignore_patterns("*.so", "*.o", "csrc", "build*", "__pycache__"))
    shutil.copy(ROOT / "sm120fp4_b200.py", tmp_path)
    (tmp_path / PKG / "libb200moe.so").symlink_to(ROOT / PKG / "libb200moe.so")
    r = subprocess.run([sys.executable, "-W", "error", "-c", code], cwd=tmp_path, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


def test_library_without_the_extension(tmp_path):
    run_without_extension(tmp_path, "import sm120fp4_b200._lib as L; assert L.host() is L.NO_HOST and L.host().quantize_own_scale(None) is None")


def test_extension_of_another_torch_is_left_out(monkeypatch):
    import sm120fp4_b200._lib as L
    assert L.host() is not L.NO_HOST and L.host().torch_version == torch.__version__
    monkeypatch.setattr(L, "_host", None)
    monkeypatch.setattr(torch, "__version__", "0.0")
    with pytest.warns(RuntimeWarning, match="built for torch"):
        assert L.host() is L.NO_HOST


def test_extension_is_built_again_for_another_torch(monkeypatch):
    spec = importlib.util.spec_from_file_location("b200moe_build_for_test", ROOT / PKG / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    assert build.HOST.name.endswith(importlib.machinery.EXTENSION_SUFFIXES[0]) and not build.host_stale()
    monkeypatch.setattr(torch, "__version__", "0.0")
    assert build.host_stale()
