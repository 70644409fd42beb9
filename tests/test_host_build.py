"""The host module belongs to one torch: it is built again for another, refused where it was built for another, and the library does without."""
import importlib.metadata
import subprocess
import sys
import types

import pytest
import torch

from jaxmodules_b200 import _native as nat, build as B


@pytest.fixture
def compiled(monkeypatch, tmp_path):
    """The compiler's command lines, in place of its runs; the module and its objects lie in a folder of their own."""
    commands = []

    def run(cmd, **_):
        commands.append(cmd)
        (tmp_path / "_host.so").write_bytes(b"")
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")

    monkeypatch.setattr(B, "HOST", tmp_path / "_host.so")
    monkeypatch.setattr(B, "OBJ", tmp_path)
    monkeypatch.setattr(subprocess, "run", run)
    return commands


def test_built_again_for_another_torch(compiled, monkeypatch):
    B._build_host(False)
    assert len(compiled) == 1 and f'-DBMA_TORCH_VERSION="{torch.__version__}"' in compiled[0]
    B._build_host(False)
    assert len(compiled) == 1
    monkeypatch.setattr(importlib.metadata, "version", lambda name: "0.0")
    B._build_host(False)
    assert len(compiled) == 2
    monkeypatch.setenv("CXX", "another-compiler")
    B._build_host(False)
    assert len(compiled) == 3 and compiled[-1][0] == "another-compiler"


def test_no_torch(compiled, monkeypatch):
    def version(name):
        raise importlib.metadata.PackageNotFoundError(name)
    monkeypatch.setattr(importlib.metadata, "version", version)
    B._build_host(True)
    assert compiled == []


def test_library_is_linked_where_the_module_fails(compiled, monkeypatch, tmp_path):
    monkeypatch.setattr(B, "LIB", tmp_path / "libbma.so")
    monkeypatch.setattr(B, "_stale", lambda *_: True)
    monkeypatch.setattr(B, "_build_host", lambda force: (_ for _ in ()).throw(RuntimeError("no host compiler")))
    with pytest.raises(RuntimeError, match="no host compiler"):
        B.build()
    assert any("-shared" in cmd and str(tmp_path / "libbma.so") in cmd for cmd in compiled)


def test_module_of_another_torch_is_refused(monkeypatch):
    fake = types.ModuleType("jaxmodules_b200._host")
    fake.torch_version = "0.0"
    monkeypatch.setattr(nat, "_host", None)
    monkeypatch.setitem(sys.modules, "jaxmodules_b200._host", fake)
    monkeypatch.setattr(sys.modules["jaxmodules_b200"], "_host", fake, raising=False)
    with pytest.raises(RuntimeError, match="built for torch 0.0"):
        nat.host()
