"""The CPython binding where there is no device: several threads in the first call, and a binding that is not built."""
import subprocess
import sys
import warnings

import pytest
import torch

import quactlize_b200 as qb
from quactlize_b200 import _lib, build

THREADS = """
import sys, threading, torch
import quactlize_b200 as qb
sys.setswitchinterval(1e-6)
b, x = torch.zeros((4, 144), dtype=torch.uint8), torch.zeros((1, 256), dtype=torch.float16)
start, got = threading.Barrier(8), []
def call():
    start.wait()
    got.append((qb._native.vecdot_dense(b, x, 4, 256, 12), qb._native.dequantize(b, 12)))   # host tensors: not served
ts = [threading.Thread(target=call) for _ in range(8)]
[t.start() for t in ts]; [t.join() for t in ts]
assert got == [(None, None)] * 8
print("ok")
"""


def test_first_call_from_several_threads():
    r = subprocess.run([sys.executable, "-c", THREADS], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]


def test_calls_work_without_the_binding(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "native_path", lambda: str(tmp_path / "absent.so"))
    absent = _lib._Native()
    monkeypatch.setattr(qb, "_native", absent)
    b = torch.zeros((4, 100), dtype=torch.uint8)
    with pytest.warns(RuntimeWarning, match="not built"):
        with pytest.raises(RuntimeError, match="144 bytes"):             # the wrapper's own check, not an ImportError
            qb.gguf_dequantize(b, 12)
    with warnings.catch_warnings():
        warnings.simplefilter("error")                                   # said once
        with pytest.raises(RuntimeError):
            qb.gguf_vecdot_rows(b, torch.zeros((1, 256), dtype=torch.float16), 4, 256, 12)
    assert absent.vecdot_moe(1, 2, 3, 4) is None


def test_a_binding_that_does_not_load_is_absent(monkeypatch, tmp_path):
    (tmp_path / "broken.so").write_bytes(b"not a shared object")
    monkeypatch.setattr(build, "native_path", lambda: str(tmp_path / "broken.so"))
    with pytest.warns(RuntimeWarning):
        assert _lib._Native().dequantize(None, 12) is None
