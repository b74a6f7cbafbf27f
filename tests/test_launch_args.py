"""The launch functions' own argument handling (csrc/py_launch.cpp), up to the C ABI's argument checks: nothing is launched."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

# A tensor of a CUDA device that has no storage, without a GPU: what a function under torch.vmap is given.
NO_STORAGE = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from qwen_engine_b200 import ops
def call(x):
    try:
        ops.launch_gemv_w4a16(x, x, x, None, x, 16, 256, stream=0)
    except RuntimeError as e:
        print("raised", type(e).__name__)
    return x
with FakeTensorMode():
    torch.vmap(call)(torch.empty(2, 256, device="cuda", dtype=torch.float16))
"""
# No stream given, and no GPU to have one (with a GPU the null weights are refused instead).
NO_STREAM = """
from qwen_engine_b200 import ops
try:
    ops.launch_gemv_w4a16(None, None, None, None, None, 16, 256)
except RuntimeError as e:
    print("raised", type(e).__name__)
"""


@pytest.mark.parametrize("script", [NO_STORAGE, NO_STREAM], ids=["no_storage", "no_stream"])
def test_errors_of_torch_are_python_errors(script):
    r = subprocess.run([sys.executable, "-W", "ignore", "-c", script], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and "raised " in r.stdout, r.stderr[-2000:]
