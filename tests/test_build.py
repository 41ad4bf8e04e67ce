"""The native build on hosts that lack something: what can be built is built."""
import sys

import pytest

from kernel_align_b200 import _build


@pytest.fixture
def elsewhere(tmp_path, monkeypatch):
    """The extension module goes to a folder of its own, and nothing is taken for built."""
    monkeypatch.setattr(_build, "LIB_DIR", tmp_path)
    monkeypatch.setattr(_build, "TORCH_LIB", tmp_path / "_ka_torch.so")
    return tmp_path


@pytest.mark.parametrize("lacks", ["torch", "headers", "torch with CUDA", "compiler", "a source that compiles"])
def test_a_host_without_what_the_autograd_module_needs(elsewhere, monkeypatch, lacks):
    import torch

    if lacks == "torch":
        monkeypatch.setitem(sys.modules, "torch", None)
    elif lacks == "headers":
        monkeypatch.setenv("CUDA_HOME", str(elsewhere))
        monkeypatch.setattr(_build, "_cuda_include", lambda: None, raising=False)
    elif lacks == "torch with CUDA":
        monkeypatch.setattr(torch.version, "cuda", None)
        monkeypatch.setattr(torch, "__file__", str(elsewhere / "torch" / "__init__.py"))
    elif lacks == "compiler":
        monkeypatch.setattr(_build.shutil, "which", lambda name: None)
    else:
        (elsewhere / "csrc" / "torch").mkdir(parents=True)
        (elsewhere / "csrc" / "torch" / "bad.cpp").write_text("#error no\n")
        monkeypatch.setattr(_build, "CSRC", elsewhere / "csrc")
        monkeypatch.setattr(_build, "ROOT", elsewhere)
    assert _build.build_torch() is None
    assert not (elsewhere / "_ka_torch.so").exists()
    if lacks != "a source that compiles":
        assert _build.torch_missing()


def test_the_kernel_library_is_built_before_the_module(monkeypatch):
    order = []
    for name in ("build_cpu", "build_cuda", "build_torch"):
        monkeypatch.setattr(_build, name, lambda *a, name=name: order.append(name))
    _build.build_all()
    assert order == ["build_cpu", "build_cuda", "build_torch"]
