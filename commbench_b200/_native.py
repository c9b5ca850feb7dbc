"""ctypes binding of ``lib/libcommbench_b200.so`` (C ABI).

The library is built in-tree by :mod:`commbench_b200._build`; importing this module never
compiles anything unless ``CB200_AUTOBUILD=1``.  On a machine with a GPU a missing
library is an error (no silent PyTorch fallback): ops that need it raise.
"""
from __future__ import annotations

import ctypes as C
import os
from pathlib import Path

MAX_RANKS = 8
PAD_CHANNELS = 1024
PAD_NVLS_BASE = PAD_CHANNELS * MAX_RANKS
PAD_ABORT = PAD_NVLS_BASE + PAD_CHANNELS
PAD_WORDS = PAD_ABORT + 64

_LIB_PATH = Path(__file__).resolve().parent / "lib" / "libcommbench_b200.so"
_FAST_PATH = _LIB_PATH.with_name("_fast_ops.so")
_lib = None
_fast = None


class NativeError(RuntimeError):
    pass


class CbComm(C.Structure):
    _fields_ = [
        ("rank", C.c_int32),
        ("world", C.c_int32),
        ("pad", C.c_void_p * MAX_RANKS),
        ("mc_pad", C.c_void_p),
        ("epoch", C.c_void_p),
        ("status", C.c_void_p),
        ("timeout_ns", C.c_uint64),
        ("jitter_ns", C.c_uint32),
        ("reserved", C.c_uint32),
    ]


class CollArgs(C.Structure):
    _fields_ = [
        ("comm", CbComm),
        ("sym", C.c_void_p * MAX_RANKS),
        ("mc", C.c_void_p),
        ("inp", C.c_void_p),
        ("out", C.c_void_p),
        ("nbytes", C.c_ulonglong),
        ("copy_in", C.c_int),
        ("copy_out", C.c_int),
        ("root", C.c_int),
        ("dtype", C.c_int),
        ("a2a_b", C.c_int),
        ("a2a_s_local", C.c_int),
        ("a2a_h", C.c_int),
        ("a2a_d", C.c_int),
        ("a2a_to_heads", C.c_int),
        ("unroll", C.c_int),
        ("variant", C.c_int),
    ]


# op codes of cb_coll_launch
OP_AR_ONESHOT, OP_AR_TWOSHOT, OP_AR_NVLS, OP_AG_PULL, OP_AG_PUSH, OP_RS, OP_A2A_FLAT, OP_A2A_4D, \
    OP_BCAST = range(9)
DT_BF16, DT_F16, DT_F32 = 0, 1, 2

STATUS_CODES = {
    0: "ok",
    1: "timeout waiting for a peer GPU's flag",
    2: "timeout on an mbarrier inside a CTA",
    3: "timeout waiting for another CTA's flag",
    4: "a peer aborted",
    5: "bad argument detected on the device",
    6: "timeout waiting for a host-written flag",
}


def decode_status(word: int) -> str:
    code, phase, detail = word >> 24, (word >> 16) & 0xFF, word & 0xFFFF
    return f"{STATUS_CODES.get(code, f'code {code}')} (phase {phase}, detail {detail})"


def lib_path() -> Path:
    return _LIB_PATH


def available() -> bool:
    return _LIB_PATH.exists()


# Entry points of the per-call operators take plain integers for pointers: declared argument types
# spare a ctypes object per argument.
_P, _I, _F, _L = C.c_void_p, C.c_int, C.c_float, C.c_longlong
_HOT_ARGTYPES = {
    "cb_gemm_bf16": [_P, _P, _P, _I, _I, _I, _F, _I, _I, _P, _P],
    "cb_gemm_fp8": [_P, _P, _P, _I, _I, _I, _F, _I, _I, _P, _P],
    "cb_gemm_small": [_P, _P, _P, _I, _I, _I, _F, _I, _I, _I, _P, _P],
    "cb_gemm_fp8_mx": [_P, _P, _P, _P, _P, _I, _I, _I, _F, _I, _P, _P],
    "cb_gemm_fp8_blockscaled": [_P, _P, _P, _P, _P, _I, _I, _I, _F, _I, _I, _P, _P],
    "cb_quant_blockscaled": [_P, _P, _P, _L, _I, _I, _P],
    "cb_quant_blockscaled_pow2": [_P, _P, _P, _P, _I, _L, _I, _I, _P],
    "cb_attn_fwd": [_P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _F, _P, _P],
    "cb_attn_fwd4": [_P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _F, _P, _P],
    "cb_attn_split_bytes": [_I, _I, _I, _I, _I, _I, _I, _I],
    "cb_attn_split": [_P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _I, _F, _P, _L, _P, _P],
    "cb_moe_router_topk": [_P, _I, _I, _I, _P, _P, _P],
    "cb_moe_slots": [_P, _I, _I, _P, _P, _P],
    "cb_moe_plan": [_P, _I, _I, _I, _P, _P, _P, _P, _P, _I, _P, _P],
}


def load():
    """Returns the loaded library, building it first only if CB200_AUTOBUILD=1."""
    global _lib
    if _lib is not None:
        return _lib
    if not _LIB_PATH.exists():
        if os.environ.get("CB200_AUTOBUILD", "0") == "1":
            from . import _build

            _build.build()
        else:
            raise NativeError(
                f"{_LIB_PATH} is missing: run `python -m commbench_b200._build` "
                "(or __graft_entry__.build()) first")
    lib = C.CDLL(str(_LIB_PATH), mode=C.RTLD_GLOBAL)
    lib.cb_last_error.restype = C.c_char_p
    for name in ("cb_symm_round_size", "cb_attn_split_bytes"):
        getattr(lib, name).restype = C.c_longlong
    for name, args in _HOT_ARGTYPES.items():
        getattr(lib, name).argtypes = args
    if lib.cb_sizeof_coll_args() != C.sizeof(CollArgs):
        raise NativeError(
            f"CollArgs layout mismatch: C {lib.cb_sizeof_coll_args()} vs ctypes {C.sizeof(CollArgs)}")
    _lib = lib
    return lib


_FAST_ENTRIES = ("cb_gemm_bf16", "cb_gemm_fp8", "cb_gemm_fp8_blockscaled", "cb_gemm_fp8_mx",
                 "cb_quant_blockscaled", "cb_quant_blockscaled_pow2", "cb_attn_fwd4",
                 "cb_attn_split_bytes", "cb_attn_split")


class _NoFast:
    """Stands in for an extension that is not there: takes no call."""

    def __getattr__(self, name):
        return lambda *args: None


def fast():
    """The extension with the short call path of the small operators (host/fast_ops.cpp).  Each of its
    functions answers None for a call that it leaves to the general path.  So do all of them, after one
    warning, where the extension is missing or was built for another PyTorch: the kernels are in the
    library that :func:`load` opens, and only the host's share of a call gets longer."""
    global _fast
    if _fast is None:
        import importlib.machinery
        import importlib.util
        import warnings

        from . import _build

        lib = load()
        try:
            if not _FAST_PATH.exists():
                raise ImportError(f"{_FAST_PATH} is missing")
            loader = importlib.machinery.ExtensionFileLoader("_fast_ops", str(_FAST_PATH))
            mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("_fast_ops", loader))
            loader.exec_module(mod)
            made_for = getattr(mod, "built_for", lambda: "an unknown PyTorch")()
            if made_for != _build.built_for():
                raise ImportError(f"{_FAST_PATH} was built for {made_for}, this is {_build.built_for()}")
            mod.bind({n: C.cast(getattr(lib, n), C.c_void_p).value for n in _FAST_ENTRIES})
            _fast = mod
        except ImportError as e:
            _fast = _NoFast()
            warnings.warn(f"short call path off ({e}); `python -m commbench_b200._build` builds it",
                          RuntimeWarning, stacklevel=2)
    return _fast


def last_error() -> str:
    lib = load()
    s = lib.cb_last_error()
    return s.decode() if s else ""


def check(rc: int, what: str) -> None:
    if rc != 0:
        raise NativeError(f"{what} failed (rc={rc}): {last_error()}")


def ptr(t) -> C.c_void_p:
    """Device pointer of a torch tensor (or None)."""
    return C.c_void_p(0 if t is None else t.data_ptr())


def raw_stream(stream=None) -> int:
    """Handle of ``stream``, or of the current stream of the current device.  The raw query costs
    0.3 us where building the ``torch.cuda.Stream`` object costs 3.5."""
    if stream is not None:
        return stream.cuda_stream
    import torch

    try:
        return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())
    except AttributeError:               # private: may be missing in another torch
        return torch.cuda.current_stream().cuda_stream


def new_empty_on(stream, like, shape, dtype=None, handed_out: bool = True):
    """``like.new_empty`` for memory that a call running on ``stream`` writes.

    It comes from the pool of the stream that writes it: a block of the current stream's pool may have
    been freed with work of that stream still queued on it, and nothing orders ``stream`` behind that
    work.  For a result (``handed_out``), the current stream, where the caller goes on with it, is
    recorded as a second user, so that the block is not reused before that stream is done either."""
    import torch

    with torch.cuda.stream(stream):
        t = like.new_empty(shape, dtype=dtype)
    if handed_out:
        t.record_stream(torch.cuda.current_stream(t.device))
    return t


def stream_ptr(stream=None) -> C.c_void_p:
    return C.c_void_p(raw_stream(stream))
