"""B200 (sm_100a) implementation of the W4A16 group-128 projection path of qwen-engine.

The product is the CUDA library `libw4a16_b200.so` behind the C ABI in
`include/w4a16_b200.h`; `ops` is a thin Python mirror of the reference's launch functions
over that ABI (torch supplies device memory and streams only).
"""
from . import _lib, ops  # noqa: F401

globals().update({_n: getattr(ops, _n) for _n in ops.__all__ if _n not in ops._NATIVE})
__all__ = [_n for _n in globals() if not _n.startswith("_")] + list(ops._NATIVE)


def __getattr__(name: str):
    # a launch function: loads the CUDA library on first use, after which it is an attribute like the others
    if name not in ops._NATIVE:
        raise AttributeError(f"module {__name__!r} has no attribute {name!r}")
    fn = getattr(ops, name)
    globals().update({n: f for n in ops._NATIVE if (f := vars(ops).get(n)) is not None})
    return fn
