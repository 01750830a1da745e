"""The compiled call path of the ops (csrc/fastops.cpp) on the host: what torch throws in it
reaches Python as an exception. In a process of its own, which an exception that nobody
catches would end."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent

# Tensors that say they are CUDA tensors and have no storage: without a device, torch throws on the
# way (no driver to ask for a stream or for memory).
SCRIPT = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from svod_b200 import _lib
fast = _lib.fastops()
with FakeTensorMode():
    t = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device="cuda")
    x, w, q, n = t(4, 64), t(32, 64), t(1, 4, 2, 64), t(64)
    for call in (lambda: fast.linear(x, w, None), lambda: fast.attention(q, q, q, None),
                 lambda: fast.attention_packed(t(1, 4, 384), 2, 2, None), lambda: fast.norm(x, None, n, None, 1e-5, True)):
        try:
            call()
        except RuntimeError:
            print("raised")
"""


@pytest.mark.skipif(torch.cuda.is_available(), reason="with a device nothing throws here")
def test_what_torch_throws_is_raised():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split() == ["raised"] * 4, (r.returncode, r.stderr[-500:])


def test_the_library_builds_and_the_ops_work_without_the_compiled_call_path(tmp_path, monkeypatch, capsys):
    from svod_b200 import _lib, build, ops
    monkeypatch.setattr(build, "FAST", tmp_path / "_fastops.so")
    monkeypatch.setattr(build, "CXX", "false")  # no headers, no compiler: whatever keeps it from being built
    build.FAST.write_bytes(b"an older build")
    assert build.build() == build.LIB
    assert not build.FAST.exists() and "_fastops.so" in capsys.readouterr().err
    # the ops then go the general way: its checks, its errors
    monkeypatch.setattr(_lib, "_fast", None)
    monkeypatch.setattr(ops, "_call", None)
    monkeypatch.setattr(_lib, "__file__", str(tmp_path / "_lib.py"))
    with pytest.warns(UserWarning, match="svod_b200.build"), pytest.raises(ops.OpsError) as e:
        ops.linear(torch.zeros(2, 4), torch.zeros(3, 4))
    assert e.value.kind == "Unrealized"


def test_another_torch_builds_the_call_path_anew(tmp_path, monkeypatch):
    from importlib import metadata
    from svod_b200 import build
    monkeypatch.setattr(build, "FAST", tmp_path / "_fastops.so")
    ran = []

    def compiler(cmd, **kw):
        ran.append(cmd)
        build.FAST.write_bytes(b"built")
        return subprocess.CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(build.subprocess, "run", compiler)
    build._build_fast()
    build._build_fast()
    assert len(ran) == 1
    monkeypatch.setattr(metadata, "version", lambda name: "0.0.1")
    build._build_fast()
    assert len(ran) == 2
