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
