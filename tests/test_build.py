"""The torch binding is built against one torch: with another it is out of date, for build.py as for whoever loads it."""
import importlib.util
import os

import pytest
import torch

from conftest import PKG_DIR
from dfa3d_b200 import _lib


@pytest.fixture
def build_py(lib_built):
    spec = importlib.util.spec_from_file_location("dfa3d_build", os.path.join(PKG_DIR, "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_another_torch_needs_a_build(build_py, monkeypatch):
    assert not build_py.needs_build()
    monkeypatch.setattr(torch, "__version__", "9.9.9+other")
    assert build_py.needs_build()


def test_binding_of_another_torch_is_not_used(build_py, monkeypatch):
    assert _lib.native() is not None
    monkeypatch.setattr(_lib, "_native", None)
    monkeypatch.setattr(torch, "__version__", "9.9.9+other")
    with pytest.raises(ImportError, match="was built for torch .* this is torch 9.9.9"):
        _lib.native()


def test_headers_come_from_the_toolkit_of_nvcc(build_py, monkeypatch, tmp_path):
    nvcc = tmp_path / "bin" / "nvcc"
    nvcc.parent.mkdir()
    nvcc.write_text("#!/bin/sh\n")
    nvcc.chmod(0o755)
    monkeypatch.setenv("NVCC", str(nvcc))
    assert os.path.join(os.path.realpath(tmp_path), "include") in build_py._native_command()
