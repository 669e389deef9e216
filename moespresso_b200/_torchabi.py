"""Glue between torch CUDA tensors and the C ABI: dtype codes, pointers, streams,
argument structures.  Torch is used for device memory and streams only."""
from __future__ import annotations

import ctypes as C
import warnings

import torch

from . import _abi

_DTYPES = {
    torch.float32: _abi.F32,
    torch.float16: _abi.F16,
    torch.bfloat16: _abi.BF16,
    torch.int8: _abi.I8,
}
if hasattr(torch, "float8_e4m3fn"):
    _DTYPES[torch.float8_e4m3fn] = _abi.F8E4M3


def dtype_code(t: torch.Tensor) -> int:
    try:
        return _DTYPES[t.dtype]
    except KeyError:
        raise ValueError(f"unsupported dtype {t.dtype}") from None


def require_cuda(*tensors) -> torch.device:
    dev = None
    for t in tensors:
        if t is None:
            continue
        if not isinstance(t, torch.Tensor) or not t.is_cuda:
            raise RuntimeError(
                "moespresso_b200 operators run on CUDA tensors only; there is no CPU path")
        if dev is None:
            dev = t.device
        elif t.device != dev:
            raise ValueError("all tensors must live on the same CUDA device")
    if dev is None:
        raise RuntimeError("moespresso_b200 operators need at least one CUDA tensor")
    return dev


def ptr(t) -> int | None:
    return None if t is None else t.data_ptr()


def stream_ptr() -> C.c_void_p:
    """The current device's current stream (the raw handle: a ``torch.cuda.Stream`` object per launch is 4 us)."""
    return C.c_void_p(torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()))


def workspace(nbytes: int, device) -> torch.Tensor | None:
    if nbytes <= 0:
        return None
    return torch.empty(int(nbytes), dtype=torch.uint8, device=device)


def status_word(device) -> torch.Tensor:
    return torch.zeros(1, dtype=torch.int32, device=device)


def last_dim_contiguous(t: torch.Tensor) -> torch.Tensor:
    return t if t.stride(-1) == 1 else t.contiguous()


# Optional per-entry-point device timing: set TIMER to a dict and every launch records a
# pair of CUDA events on the current stream around the C call (name -> [(start, end), ...]).
TIMER = None


_NATIVE_CALLS = ("mxb_indexer_scores", "mxb_topk_workspace_bytes", "mxb_topk_select", "mxb_sparse_attn_workspace_bytes",
                 "mxb_sparse_attn", "mxb_fused_decode_prep_workspace_bytes", "mxb_fused_decode_prep",
                 "mxb_fused_decode_sdpa_workspace_bytes", "mxb_fused_decode_sdpa", "mxb_affine_q8_append",
                 "mxb_sdpa_decode_q8", "mxb_merge_partials")
_native = None     # the extension; False: there is none, every call is the Python operators'


def _load_native():
    """The CPython extension, built first where it is missing or belongs to another torch or interpreter (loaded all the
    same it would misread their objects).  Where that cannot be done the Python operators take every call, at their own pace."""
    from . import _build
    lib = _abi.load()
    try:
        if not _build.native_is_current():
            _build.build_native()
        from . import _native as mod
        mod.bind(*(C.cast(getattr(lib, n), C.c_void_p).value for n in _NATIVE_CALLS))
        return mod
    except (ImportError, OSError, RuntimeError) as e:
        warnings.warn(f"moespresso_b200: no native host calls, short steps run from Python and take longer ({e})", RuntimeWarning,
                      stacklevel=4)
        return False


def native(name: str, *args):
    """One of the native host calls (``csrc/host_calls.cpp``), which take an operator's plain case in one go.  None: not
    such a case, the caller goes on in Python."""
    global _native
    if _native is None:
        _native = _load_native()
    if TIMER is not None or _native is False:
        return None
    r = getattr(_native, name)(*args)
    if type(r) is int:
        _abi.check(r)
    return r


def launch(name: str, fn, args) -> int:
    if TIMER is None:
        return fn(C.byref(args), stream_ptr())
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    rc = fn(C.byref(args), stream_ptr())
    e1.record()
    TIMER.setdefault(name, []).append((e0, e1))
    return rc
