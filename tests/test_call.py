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


def test_the_library_builds_without_torch(monkeypatch):
    from zinc_b200 import build

    monkeypatch.setattr(build, "_torch_spec", lambda: None)
    assert build._call_command() is None   # nothing to compile beside the library, no error


def test_without_the_native_module_calls_go_through_ctypes():
    r = run("""
import sys
sys.modules["zinc_b200._call"] = None   # as where it was not built
import torch
from zinc_b200 import dispatch
f = dispatch._calls()
assert f["zc_dmmv"].__module__ == "zinc_b200.dispatch"
print(f["zc_bias_add"](0, dispatch.Buffer(None, 0), dispatch.Buffer(None, 0), 4, 0))
""")
    assert r.returncode == 0 and r.stdout.split() == ["3"], r.stderr[-500:]


@pytest.mark.parametrize("native", [True, False])
def test_arguments_arrive(native):
    """Every function of the table is entered with its own signature: a callee of the declared types sees the values."""
    r = run(f"""
import ctypes as C, sys
{'import torch' if native else ''}
from zinc_b200 import _lib, dispatch
L = _lib.lib()
seen = []
class Fake:      # functions of the exported ones' types that note what they get
    pass
keep = []
for name in dispatch._CALLS:
    args = getattr(L, name).argtypes
    cb = C.CFUNCTYPE(C.c_int32, *args)(lambda *a: seen.append(a) or 7)
    cb.argtypes = args
    keep.append(cb)
    setattr(Fake, name, cb)
_lib.lib = lambda: Fake
calls = dispatch._calls()
assert (type(calls['zc_dmmv']).__name__ == 'Call') == {native}
for name, spec in dispatch._CALLS.items():
    given, want, n = [], [], 0
    for kind in spec:
        n += 1
        if kind == 'f':
            given.append(0.5); want.append(0.5)
        elif kind == 'i':
            given.append(1000 + n); want.append(1000 + n)
        elif kind == 'o' and n % 2:
            given.append(None); want += [None, 0]
        else:
            given.append(dispatch.Buffer(4096 * n, 16 * n)); want += [4096 * n, 16 * n]
    assert calls[name](*given) == 7, name
    assert list(seen.pop()) == want, name
big = (1 << 40) + 8   # byte offsets are 64 bits wide
calls['zc_dmmv'](1, 12, *[dispatch.Buffer(64, big)] * 3, 5, 6, big, big, big, 1)
assert seen.pop()[7:] == (big, 5, 6, big, big, big, 1)
print('ok')
""")
    assert r.returncode == 0 and r.stdout.split() == ["ok"], r.stderr[-800:]
