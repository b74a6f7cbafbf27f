"""The launch functions' own argument handling (csrc/py_launch.cpp), up to the C ABI's argument checks: nothing is launched."""
import ctypes
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


class Device:
    """Stands in for a tensor on the GPU."""
    is_cuda = True

    def __init__(self, address=256):
        self.address = address

    def data_ptr(self):
        return self.address


class Stream:
    cuda_stream = 0


class Number:
    def __init__(self, value):
        self.value = value

    def __index__(self):
        return self.value


def _gemv(**changes):
    """launch_gemv_w4a16 up to the C ABI, which refuses K = 100."""
    from qwen_engine_b200 import ops
    d = Device()
    args = dict(qweight=d, scales=d, input_x=d, residual=None, output_y=d, out_features=16, in_features=100, stream=0)
    args.update(changes)
    return ops.launch_gemv_w4a16(**args)


def _status(call):
    from qwen_engine_b200 import ops
    with pytest.raises(ops.W4A16Error) as e:
        call()
    return e.value.status


def test_arguments_reach_the_c_function_by_position_and_by_name():
    from qwen_engine_b200 import ops
    d = Device()
    assert _status(_gemv) == -2                                                        # all by name
    assert _status(lambda: ops.launch_gemv_w4a16(d, d, d, None, d, 16, 100, 0)) == -2  # all by position
    assert _status(lambda: ops.launch_gemv_w4a16(d, d, d, in_features=100, residual=None, output_y=d, out_features=16, stream=0)) == -2
    assert _status(lambda: _gemv(output_y=None)) == -1
    assert _status(lambda: _gemv(in_features=256, output_y=Device(257))) == -3
    assert _status(lambda: _gemv(out_features=Number(16), in_features=Number(100))) == -2
    assert _status(lambda: _gemv(out_features=True, in_features=False)) == -2
    # defaults of what is left out: 1536 is a multiple of 128, the address is not one of 8
    assert _status(lambda: ops.launch_rmsnorm_q8_1(Device(2), d, None, d, d, d, 0)) == -3
    assert _status(lambda: ops.launch_rmsnorm_q8_1(d, d, None, d, d, d, 0, 100)) == -2


@pytest.mark.parametrize("args,kwargs,error,text", [
    ((1,) * 9, {}, TypeError, "at most 8 arguments"),
    ((None,) * 7, {"nothing": 1}, TypeError, "unexpected keyword argument 'nothing'"),
    ((None,) * 7, {"scales": 1}, TypeError, "multiple values for argument 'scales'"),
    ((None,) * 6, {}, TypeError, "missing required argument 'in_features'"),
    ((), {"qweight": None}, TypeError, "missing required argument 'scales'"),
    ((None,) * 5 + (1 << 31, 256, 0), {}, OverflowError, "C int"),
    ((None,) * 5 + (16, -(1 << 31) - 1, 0), {}, OverflowError, "C int"),
    ((None,) * 5 + (1 << 80, 256, 0), {}, OverflowError, None),
    ((None,) * 5 + (16.0, 256, 0), {}, TypeError, None),
    ((None,) * 5 + ("16", 256, 0), {}, TypeError, None),
    ((None,) * 5 + (16, 256, "stream"), {}, ValueError, None),
    ((None,) * 5 + (16, 256, object()), {}, TypeError, None),
    ((None,) * 5 + (16, 256, 1 << 80), {}, OverflowError, None),
    ((256,) + (None,) * 4 + (16, 256, 0), {}, AttributeError, "is_cuda"),      # an address is no tensor
])
def test_wrong_arguments(args, kwargs, error, text):
    from qwen_engine_b200 import ops
    with pytest.raises(error, match=text):
        ops.launch_gemv_w4a16(*args, **kwargs)


def test_tensors_off_the_device_are_refused():
    import torch
    from qwen_engine_b200 import ops
    for where in ("cpu", "meta"):
        t = torch.empty(256, dtype=torch.float16, device=where)
        with pytest.raises(ValueError, match="not on a CUDA device"):
            _gemv(input_x=t)
        with pytest.raises(ValueError, match="not on a CUDA device"):
            ops.launch_gemv_qkv_w4a8(ops.QKVProjectionView(*[Device()] * 8, t), Device(), Device(), Device(), 0)
    with pytest.raises(AttributeError, match="q_weight"):
        ops.launch_gemv_qkv_w4a8(None, Device(), Device(), Device(), 0)


def test_kinds_of_stream_without_a_launch():
    handle = type("Handle", (), {"__int__": lambda self: 0})()
    for stream in (Stream(), 0, handle, 0.0):       # an object that has a handle, and what int() takes
        assert _status(lambda stream=stream: _gemv(stream=stream)) == -2


def test_the_c_struct_of_a_view():
    """For hosts that call the C functions through load()."""
    from qwen_engine_b200 import ops
    pod = ops.QKVProjectionView(*[Device(16 * (i + 1)) for i in range(9)]).pod()
    assert [getattr(pod, n) for n, _ in pod._fields_] == [16 * (i + 1) for i in range(9)]
    d = ctypes.c_void_p(256)
    assert ops.load().w4a16_gemv_qkv_w4a8(ctypes.byref(pod), d, d, d, None, 100, 1, 1, 128) == -2


@pytest.mark.gpu
def test_kinds_of_stream_launch_where_they_say():
    """The stream object, its handle and the current stream: all three are captured, none runs outside the graph."""
    import torch
    import numpy as np
    from qwen_engine_b200 import ops, synth
    from tests import util
    N, K = 64, 256
    w, sc, x = (util.to_dev(a) for a in (synth.packed_weights(1, "s", N, K), synth.scales(1, "s", N, K), synth.activations(1, "s", K)))
    want = torch.empty(N, dtype=torch.float16, device="cuda")
    ops.launch_gemv_w4a16(w, sc, x, None, want, N, K)
    y = torch.full((3, N), float("nan"), dtype=torch.float16, device="cuda")
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        ops.launch_gemv_w4a16(w, sc, x, None, y[0], N, K, s)
        ops.launch_gemv_w4a16(w, sc, x, None, y[1], N, K, stream=s.cuda_stream)
        ops.launch_gemv_w4a16(w, sc, x, None, y[2], N, K)
    torch.cuda.synchronize()
    assert np.isnan(util.to_np(y)).all()
    graph.replay()
    torch.cuda.synchronize()
    for row in y:
        assert torch.equal(row.view(torch.int16), want.view(torch.int16))


@pytest.mark.gpu
def test_a_tensor_without_storage_is_refused_on_the_gpu():
    import torch
    from qwen_engine_b200 import ops

    def call(x):
        with pytest.raises(RuntimeError):
            ops.launch_gemv_w4a16(x, x, x, None, x, 16, 256)
        return x

    torch.vmap(call)(torch.zeros(2, 256, dtype=torch.float16, device="cuda"))
