"""The host extension is built for one torch, one interpreter and one command, and built again when any of them differs."""
import subprocess
import sysconfig
from types import SimpleNamespace

import torch

from bitnet_nvfp4_b200 import build


def test_rebuilt_when_torch_or_the_command_changes(tmp_path, monkeypatch):
    calls = []

    def run(cmd, **kw):
        calls.append(cmd)
        build.HOST.write_bytes(b"")
        return SimpleNamespace(returncode=0, stdout="", stderr="")

    monkeypatch.setattr(build, "HOST", tmp_path / "_host.so")
    monkeypatch.setattr(build, "OBJ", tmp_path / "obj")
    monkeypatch.setattr(build, "PKG", tmp_path)
    monkeypatch.setattr(subprocess, "run", run)
    build.build_host()
    build.build_host()
    assert len(calls) == 1
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", torch.__version__ + "x")
        build.build_host()
        build.build_host()
    assert len(calls) == 2
    build.build_host()
    assert len(calls) == 3
    monkeypatch.setattr(torch._C, "_GLIBCXX_USE_CXX11_ABI", not torch._C._GLIBCXX_USE_CXX11_ABI)
    build.build_host()
    assert len(calls) == 4


def test_the_file_names_its_interpreter():
    assert build.HOST.name == "_host" + sysconfig.get_config_var("EXT_SUFFIX")
