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


# Which of the package's two libraries a process has mapped.
MAPPED = """
import sys
def mapped():
    return sorted({n for l in open("/proc/self/maps") for n in ("_launch.so", "libw4a16_b200.so") if l.rstrip().endswith("/" + n)})
"""


def _python(script):
    r = subprocess.run([sys.executable, "-W", "ignore", "-c", MAPPED + script], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.split()


def test_the_cuda_library_is_loaded_by_the_first_launch_function():
    """The CPU arm of the benchmark and whoever wants shapes and synthetic tensors only stay free of it."""
    out = _python("""
from qwen_engine_b200 import nsplit, ops, qwenbin, synth
import qwen_engine_b200 as q
assert mapped() == [], mapped()
assert hasattr(q, "launch_gemv_w4a8") and q.launch_gemv_w4a8 is ops.launch_gemv_w4a8
assert mapped() == ["_launch.so", "libw4a16_b200.so"], mapped()
assert "launch_gemv_w4a8" in vars(ops) and "launch_gemm_prefill_w4a16" in vars(q)
names = {}
exec("from qwen_engine_b200 import *", names)
assert set(ops.__all__) <= set(names) and "ops" in names
assert not hasattr(ops, "launch_nothing") and not hasattr(q, "launch_nothing")
print("ok")
""")
    assert out == ["ok"]


def test_a_missing_build_says_so_when_a_function_is_called():
    out = _python("""
sys.modules["qwen_engine_b200._launch"] = None
import qwen_engine_b200 as q
f = q.launch_gemv_w4a16
try:
    f()
except ImportError as e:
    print("build" in str(e))
""")
    assert out == ["True"]


def test_the_module_is_built_anew_for_another_torch_or_python(monkeypatch):
    from qwen_engine_b200 import build
    build.build()
    assert build.up_to_date()
    for text in ("torch 2.11", "torch 0.0.1, cpython-312"):
        monkeypatch.setattr(build, "_built_for", lambda text=text: text)
        assert not build.up_to_date()
