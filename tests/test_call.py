"""The native calls of dispatch.py (csrc/call.cpp): what they take, and what they do with what they cannot take."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run(code):
    return subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)


@pytest.mark.parametrize("transform", ["torch.vmap(call)(torch.empty(2, 16, device='cuda:0'))",
                                       "torch.func.jvp(call, (torch.empty(16, device='cuda:0'),), (torch.empty(16, device='cuda:0'),))",
                                       "torch.func.vjp(call, torch.empty(16, device='cuda:0'))"])
def test_a_tensor_without_memory_raises(transform):
    # such tensors answer data_ptr() with a C++ exception: it has to arrive as a Python one and not end the process
    r = run(f"""
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from zinc_b200 import dispatch
bias_add = dispatch._calls()["zc_bias_add"]
def call(a):
    try:
        bias_add(0, a, a, 16, 0)
    except RuntimeError:
        print("raised")
    return a
with FakeTensorMode():
    {transform}
""")
    assert r.returncode == 0 and r.stdout.split() == ["raised"], (r.returncode, r.stdout, r.stderr[-500:])
