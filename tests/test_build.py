"""The native build on hosts that lack something: what can be built is built."""
import sys

import pytest

from kernel_align_b200 import _build


@pytest.fixture
def elsewhere(tmp_path, monkeypatch):
    """The extension module goes to a folder of its own, and nothing is taken for built."""
    monkeypatch.setattr(_build, "LIB_DIR", tmp_path)
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
    assert not [p for p in elsewhere.iterdir() if p.suffix in (".so", ".part", ".hash")]
    if lacks != "a source that compiles":
        assert _build.torch_missing()


def test_a_module_of_another_torch_or_of_other_sources_is_not_loaded(elsewhere, monkeypatch):
    import torch

    (elsewhere / "csrc" / "torch").mkdir(parents=True)
    monkeypatch.setattr(_build, "CSRC", elsewhere / "csrc")                # an installed package: no sources
    mine = _build.torch_lib()
    mine.write_bytes(b"")
    assert _build.build_torch() == mine
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "2.99.0")
        assert _build.torch_lib() != mine and _build.build_torch() is None
    (elsewhere / "csrc" / "torch" / "node.cpp").write_text("")             # a checkout whose module is older than its sources
    monkeypatch.setattr(_build, "ROOT", elsewhere)
    monkeypatch.setattr(_build, "torch_missing", lambda: "no compiler")
    assert _build.build_torch() is None


def test_an_installed_package_compiles_the_module_when_it_is_told_to(tmp_path, monkeypatch):
    root = tmp_path / "site"
    package = root / "kernel_align_b200"
    (package / "_src").mkdir(parents=True)
    (package / "_src" / "node.cpp").write_text("")
    for name, value in (("ROOT", root), ("CSRC", root / "csrc"), ("LIB_DIR", package / "_lib")):
        monkeypatch.setattr(_build, name, value)
    compiled = []

    def run(cmd):
        compiled.append(cmd)
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write("module")

    monkeypatch.setattr(_build, "_run", run)
    assert _build.build_torch() is None and not compiled                  # as the first call of an operator does
    path = _build.build_torch(installed=True)
    assert path.read_text() == "module" and str(package / "_src" / "node.cpp") in compiled[0]
    assert _build.build_torch() == path and _build.build_torch(installed=True) == path and len(compiled) == 1


def test_ranks_that_build_at_once_find_a_whole_module(elsewhere, monkeypatch):
    """The compiler writes beside the module, which is put in place when it is whole."""
    seen = []

    def run(cmd):
        out = cmd[cmd.index("-o") + 1]
        seen.append((out, _build.torch_lib().exists()))
        with open(out, "w") as f:
            f.write("whole")

    monkeypatch.setattr(_build, "_run", run)
    path = _build.build_torch()
    assert seen == [(seen[0][0], False)] and seen[0][0] != str(path) and path.read_text() == "whole"


def test_the_kernel_library_is_built_before_the_module(monkeypatch):
    order = []
    for name in ("build_cpu", "build_cuda", "build_torch"):
        monkeypatch.setattr(_build, name, lambda *a, name=name, **k: order.append(name))
    _build.build_all()
    assert order == ["build_cpu", "build_cuda", "build_torch"]
