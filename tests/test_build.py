"""The build without a GPU: the library needs no PyTorch, and the binding is built anew for another PyTorch."""
import importlib.util
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture
def build(tmp_path):
    """``build.py`` by itself, with one small source and its outputs in a folder of the test's own."""
    spec = importlib.util.spec_from_file_location("build_alone", ROOT / "workloadsuite_b200" / "build.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    src = tmp_path / "small.cu"
    src.write_text('extern "C" int small() { return 7; }\n')
    mod.sources = lambda: [src]
    mod.LIB_DIR = tmp_path
    for name in ("LIB", "TORCH_LIB", "STAMP", "TORCH_STAMP"):
        setattr(mod, name, tmp_path / getattr(mod, name).name)
    return mod


def test_the_library_is_built_without_pytorch(build, monkeypatch):
    monkeypatch.setitem(sys.modules, "torch", None)
    assert build.build() == build.LIB and build.LIB.exists() and not build.TORCH_LIB.exists()
    assert build.is_current()


def test_a_binding_that_does_not_compile_leaves_the_library(build, monkeypatch):
    monkeypatch.setenv("CXX", "false")
    with pytest.raises(RuntimeError):
        build.build()
    assert build.LIB.exists() and not build.is_current()
    monkeypatch.setitem(sys.modules, "torch", None)
    assert build.is_current()


def test_another_pytorch_makes_the_binding_stale(build, monkeypatch):
    import torch

    monkeypatch.setenv("CXX", "true")          # (what is compiled does not matter here)
    build.TORCH_LIB.touch()
    build.build()
    assert build.is_current()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".other")
    assert not build.is_current()
