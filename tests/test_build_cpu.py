"""The build: the C-ABI library stands without torch, the CPython binding is named after what it was compiled against."""
import importlib.util
import os
import sysconfig

import pytest
import torch

from quactlize_b200 import build


def test_binding_is_named_after_python_and_torch(monkeypatch):
    path = build.native_path()
    assert sysconfig.get_config_var("SOABI") in path and torch.__version__ in path and path.endswith(".so")
    assert os.path.exists(path)
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert build.native_path() != path and not os.path.exists(build.native_path())


def test_library_is_built_where_there_is_no_torch(monkeypatch, tmp_path):
    """Nothing of the binding is touched, and the library is linked before the binding could fail."""
    order = []
    monkeypatch.setattr(build, "LIB", str(tmp_path / "lib.so"))
    monkeypatch.setattr(build, "OBJ", str(tmp_path))
    monkeypatch.setattr(build, "sources", lambda: [])
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: order.append(cmd[0]) or type("R", (), {"returncode": 0, "stdout": "", "stderr": ""})())
    find = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    assert build.build() == build.LIB
    assert order == [build.NVCC]
    monkeypatch.undo()


def test_a_failing_binding_leaves_the_library(monkeypatch, tmp_path):
    lib = tmp_path / "lib.so"
    monkeypatch.setattr(build, "LIB", str(lib))
    monkeypatch.setattr(build, "OBJ", str(tmp_path))
    monkeypatch.setattr(build, "sources", lambda: [])

    def failing(*a):
        raise RuntimeError("g++ failed")
    monkeypatch.setattr(build, "build_native", failing)
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: lib.write_text("") or type("R", (), {"returncode": 0, "stdout": "", "stderr": ""})())
    with pytest.raises(RuntimeError, match="g.. failed"):
        build.build()
    assert lib.exists()
