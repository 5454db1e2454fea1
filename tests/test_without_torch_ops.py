"""CPU: what there is without a CUDA build of torch: the library and its bindings build, and the autograd entry points take the Python
way."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from aotriton_b200 import build

ROOT = Path(__file__).resolve().parent.parent


def test_build_leaves_the_native_route_out(monkeypatch):
    ran = []
    monkeypatch.setattr(build, "_run", lambda cmd: ran.append(cmd))
    monkeypatch.setattr(build, "build_library", lambda verbose=False: ran.append("library"))
    monkeypatch.setattr(build, "build_pymodule", lambda: ran.append("pymodule"))
    monkeypatch.setattr(torch.version, "cuda", None)
    build.build_all()
    assert ran == ["library", "pymodule"]
    monkeypatch.setitem(sys.modules, "torch", None)      # (import torch raises ImportError)
    assert build.build_torch_ops() is None


@pytest.mark.parametrize("torch_cuda", ["None", "'12.8'"])
def test_entry_points_without_the_module(torch_cuda):
    code = f"""
import sys, warnings
sys.modules["_torch_ops"] = None      # (its import raises ImportError)
import torch
torch.version.cuda = {torch_cuda}
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    from aotriton_b200 import autograd
assert [w.category for w in seen if "_torch_ops" in str(w.message)] == ([RuntimeWarning] if torch.version.cuda else [])
q, k, v = (torch.randn(1, 2, 4, 8, dtype=torch.float16, requires_grad=True) for _ in range(3))
assert autograd._attend(q, k, v, None, None, None, 0, 0, 1.0, 0.0, False, False, 1, 2, False) is None
assert autograd.last_bwd_family == 0
calls = []
autograd._Attention.apply = lambda *a: calls.append(a) or q
autograd.attention(q, k, v)
assert len(calls) == 1
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
