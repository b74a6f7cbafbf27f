"""Builds libw4a16_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and beside it the Python
entry points of the launch functions (_launch.so, host C++ on torch's headers).

    python -m qwen_engine_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libw4a16_b200.so"
LAUNCH = PKG / "_launch.so"
LAUNCH_SOURCE = CSRC / "py_launch.cpp"
SOURCES = ["c_abi.cu", "q8_1_quantize.cu", "gemv_decode.cu", "gemm_prefill.cu", "gemm_tc.cu", "decode_sweep.cu", "sweep_persistent.cu",
           "gemv_static_scratch.cu", "sampling.cu", "embed_lookup.cu", "qwenbin.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++20", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "-shared",
]


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found: the CUDA library cannot be built")
    return exe


def _inputs():
    files = [CSRC / s for s in SOURCES]
    files += sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.hpp"))
    files += [PKG.parent / "include" / "w4a16_b200.h"]
    return files


def _newer(target: Path, inputs) -> bool:
    if not target.exists():
        return False
    t = target.stat().st_mtime
    return all(f.stat().st_mtime <= t for f in inputs)


def up_to_date() -> bool:
    return _newer(LIB, _inputs()) and _launch_up_to_date()


def _built_for() -> str:
    """What the Python module depends on beside its sources: torch's C++ ABI and the interpreter's."""
    from importlib.metadata import version
    return f"torch {version('torch')}, {sys.implementation.cache_tag}"


def _launch_up_to_date() -> bool:
    # (the module carries the text in itself)
    return _newer(LAUNCH, [LAUNCH_SOURCE, PKG.parent / "include" / "w4a16_b200.h"]) and f"[{_built_for()}]".encode() in LAUNCH.read_bytes()


def build_launch(force: bool = False) -> Path:
    """The CPython module; it finds libw4a16_b200.so beside itself at run time."""
    if not force and _launch_up_to_date():
        return LAUNCH
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    torch_lib = Path(torch.__file__).resolve().parent / "lib"
    includes = [*cpp_extension.include_paths(device_type="cuda"), sysconfig.get_paths()["include"]]
    cmd = [shutil.which("g++") or "g++", "-O2", "-std=c++20", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f'-DW4_BUILT_FOR="{_built_for()}"', *[f"-isystem{p}" for p in includes],
           str(LAUNCH_SOURCE), "-o", str(LAUNCH), f"-L{PKG}", "-l:libw4a16_b200.so", f"-L{torch_lib}", "-ltorch_python",
           "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("g++ failed building _launch.so")
    return LAUNCH


def build(force: bool = False, verbose: bool = False) -> Path:
    """One nvcc -c per source file, in parallel, then one link step; then the Python module."""
    if force or not _newer(LIB, _inputs()):
        _build_lib(verbose)
    build_launch(force)
    return LIB


def _build_lib(verbose: bool) -> None:
    from concurrent.futures import ThreadPoolExecutor
    objdir = PKG / "build"
    objdir.mkdir(exist_ok=True)
    flags = [f for f in NVCC_FLAGS if f != "-shared"]
    if verbose:
        flags += ["-Xptxas", "-v"]

    def compile_one(src: str):
        obj = objdir / (Path(src).stem + ".o")
        res = subprocess.run([nvcc(), *flags, "-c", str(CSRC / src), "-o", str(obj)], cwd=str(CSRC),
                             capture_output=True, text=True)
        return src, obj, res

    with ThreadPoolExecutor(max_workers=min(len(SOURCES), os.cpu_count() or 4)) as pool:
        results = list(pool.map(compile_one, SOURCES))
    failed = False
    for src, _, res in results:
        if verbose or res.returncode != 0:
            sys.stderr.write(f"---- {src}\n" + res.stdout + res.stderr)
        failed = failed or res.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed building libw4a16_b200.so")
    link = subprocess.run([nvcc(), *NVCC_FLAGS, "-o", str(LIB), *[str(o) for _, o, _ in results]],
                          capture_output=True, text=True)
    if link.returncode != 0:
        sys.stderr.write(link.stdout + link.stderr)
        raise RuntimeError("linking libw4a16_b200.so failed")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
