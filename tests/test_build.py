"""The extension of the eager calls is an extra: the library is built without it, and it is bound only beside the torch
that it was compiled against."""

import ctypes
import importlib.util
import sys
from pathlib import Path

import pytest
import torch

from fdk import native

BUILD = Path(__file__).resolve().parents[1] / "fused-dequantisation-kernels_b200" / "build.py"


@pytest.fixture
def build(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("fdk_b200_build_under_test", BUILD)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    source = tmp_path / "csrc"
    source.mkdir()
    (source / "abi.cu").write_text("")
    (source / "eager_calls.cpp").write_text("")
    (source / "some.cuh").write_text("")
    for name, value in (("CSRC", source), ("OBJ", source / "build"), ("LIB", tmp_path / "lib.so"), ("EAGER", tmp_path / "_eager.so")):
        monkeypatch.setattr(module, name, value)
    ran = []

    def run(cmd, check):
        ran.append(cmd)
        Path(cmd[cmd.index("-o") + 1]).write_text("built")

    monkeypatch.setattr(module.subprocess, "run", run)
    module.ran = ran
    return module


def test_the_library_is_built_without_torch(build, monkeypatch, capsys):
    monkeypatch.setitem(sys.modules, "torch", None)  # an import of it fails
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None)
    assert build.build() == build.LIB and build.LIB.exists() and not build.EAGER.exists()
    assert "eager calls go through Python" in capsys.readouterr().err


def test_the_library_is_built_where_the_extension_does_not_compile(build, monkeypatch):
    good = build.subprocess.run

    def run(cmd, check):
        if str(build.EAGER) in cmd:
            raise build.subprocess.CalledProcessError(1, cmd)
        good(cmd, check)

    monkeypatch.setattr(build.subprocess, "run", run)
    build.EAGER.write_text("an older one")
    assert build.build(force=True).exists() and not build.EAGER.exists()


def test_another_torch_makes_another_extension(build, monkeypatch):
    build.build()
    first = len(build.ran)
    build.build()
    assert build.EAGER.exists() and len(build.ran) == first
    monkeypatch.setattr(torch, "__version__", "1.0")
    build.build()
    assert len(build.ran) == first + 1 and str(build.EAGER) in build.ran[-1]


def test_the_extension_of_another_torch_is_not_bound(monkeypatch):
    from fdk import _eager

    handle = native.lib()
    names = ("eager_linear", "eager_quantise", "eager_repack")
    for version, bound in ((str(torch.__version__), True), ("1.0", False)):
        monkeypatch.setattr(_eager, "torch_version", version, raising=False)
        for name in names:
            monkeypatch.setattr(native, name, native._nothing)
        native._bind_eager(handle)
        assert all((getattr(native, name) is not native._nothing) == bound for name in names)
    assert isinstance(handle, ctypes.CDLL)
