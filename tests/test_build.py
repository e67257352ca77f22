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


def _report(source, kernel, numbers):
    """What ptxas reported of the one kernel whose mangled name holds `kernel` when `source` was compiled: the numbers that the
    expression `numbers` finds."""
    import re
    log = os.path.join(PKG_DIR, "build", source + ".log")
    if not os.path.exists(log):
        pytest.skip("the library was not compiled here")
    with open(log) as f:
        text = f.read()
    found = re.findall(r"Compiling entry function '\S*%s\S*' .*?%s" % (re.escape(kernel), numbers), text, re.S)
    assert len(found) == 1, (kernel, found)
    return sum(int(x) for x in ([found[0]] if isinstance(found[0], str) else found[0]))


def _spill_bytes(build_py, source, kernel):
    return _report(source, kernel, r"(\d+) bytes spill stores, (\d+) bytes spill loads")


# A launch of full size walks its groups of items with a constant bound: as a run-time number it cost these kernels registers
# and up to 3 % (16-bit rows without scores 32 bytes, now 16; fp32 rows of 64 channels 68, now 36).
@pytest.mark.parametrize("source,kernel,most", [
    ("dfa3d_forward.cu", "dfa3d_forward_kernelI13__nv_bfloat16S1_Li32ELi0ELb0ELb1ELi8E", 16),
    ("dfa3d_forward.cu", "dfa3d_forward_kernelI6__halfS1_Li32ELi0ELb0ELb1ELi8E", 16),
    ("dfa3d_forward.cu", "dfa3d_forward_kernelIffLi64ELi0ELb0ELb1ELi8E", 36),
    ("dfa3d_backward.cu", "dfa3d_backward_kernelI13__nv_bfloat16S1_Li32ELi2ELb1ELi4E", 140),
    ("dfa3d_backward.cu", "dfa3d_backward_kernelIf13__nv_bfloat16Li32ELi2ELb1ELi4E", 152)])
def test_full_size_launches_have_a_constant_walk(build_py, source, kernel, most):
    assert _spill_bytes(build_py, source, kernel) <= most


# Several items a warp: fp32 rows keep their way of adding partial sums up where the 16-bit one's costs registers (2-D from
# offsets, 4 points of 32 channels 44 bytes, now none; 16 points of 16 channels with scores 36, now none).
@pytest.mark.parametrize("kernel", ["IffLi32ELi3ELb0ELi4ELb1E", "IffLi64ELi3ELb0ELi8ELb1E", "IffLi16ELi0ELb1ELi16ELb1E"])
def test_fp32_items_that_share_a_warp_spill_nothing(build_py, kernel):
    assert _spill_bytes(build_py, "dfa3d_forward_packed.cu", "dfa3d_forward_packed_kernel" + kernel) == 0


# Registers of 256 threads and with them the CTAs on an SM.  Distribution producer, backward: rows of 16-bit gradients that were
# widened when they came took 76 registers for 65 to 128 bins (three CTAs, now four).  Forward of more than 128 bins: 75 to 80.
@pytest.mark.parametrize("words", ["Li2ELi8E", "Li4ELi4E", "Li1ELi16E"])
@pytest.mark.parametrize("dtype", ["13__nv_bfloat16", "6__half"])
def test_four_ctas_of_the_16_bit_producer_backward(dtype, words):
    assert _report("dfa3d_dist_producer.cu", "32dist_from_logits_backward_kernelI" + dtype + words, r"Used (\d+) registers") <= 64


@pytest.mark.parametrize("words", ["Li1ELi32E", "Li2ELi16E", "Li4ELi8E"])
@pytest.mark.parametrize("dtype", ["f", "13__nv_bfloat16", "6__half"])
def test_four_ctas_of_the_producer_forward_of_many_bins(dtype, words):
    assert _report("dfa3d_dist_producer.cu", "23dist_from_logits_kernelI" + dtype + words, r"Used (\d+) registers") <= 64
