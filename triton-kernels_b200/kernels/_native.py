"""ctypes binding of ``libb200attn.so`` (the C ABI declared in ``include/b200attn.h``).

The library holds sm_100a code only.  There is no fallback of any kind: if the
shared object is missing or a call fails, a ``RuntimeError`` carrying the
library's own error text is raised.
"""
from __future__ import annotations

import ctypes as C
import os
import threading
import warnings
from typing import Dict, Optional, Tuple

import torch

ABI_VERSION = 1

F16, BF16, F32 = 0, 1, 2
DENSE, RAGGED, PAGED = 0, 1, 2

DTYPE_CODE = {torch.float16: F16, torch.bfloat16: BF16, torch.float32: F32}

_LIB_NAME = "libb200attn.so"
_PKG_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

EXPORTS = (
    "b200attn_abi_version",
    "b200attn_last_error",
    "b200attn_device_info",
    "b200attn_prefill_workspace_bytes",
    "b200attn_decode_workspace_bytes",
    "b200attn_decode_route",
    "b200attn_decode_keys_as_rows",
    "b200attn_prefill_route",
    "b200attn_prefill",
    "b200attn_decode",
    "b200attn_decode_static",
    "b200attn_decode_static_check",
    "b200attn_selftest_wait_expiry",
    "b200attn_selftest_cluster_expiry",
    "b200attn_selftest_abandoned_units",
    "b200attn_paged_append",
    "b200attn_softmax",
    "b200attn_check_workspace",
)


class DeviceInfo(C.Structure):
    _fields_ = [
        ("sm_count", C.c_int32),
        ("cc_major", C.c_int32),
        ("cc_minor", C.c_int32),
        ("max_smem_optin", C.c_int32),
    ]


class PrefillArgs(C.Structure):
    _fields_ = [
        ("q", C.c_void_p),
        ("k", C.c_void_p),
        ("v", C.c_void_p),
        ("out", C.c_void_p),
        ("q_indptr", C.c_void_p),
        ("kv_indptr", C.c_void_p),
        ("k_table", C.c_void_p),
        ("v_table", C.c_void_p),
        ("workspace", C.c_void_p),
        ("workspace_bytes", C.c_size_t),
        ("total_q", C.c_int64),
        ("total_kv", C.c_int64),
        ("table_stride", C.c_int64),
        ("dtype", C.c_int32),
        ("layout", C.c_int32),
        ("indptr_is_i64", C.c_int32),
        ("batch", C.c_int32),
        ("q_heads", C.c_int32),
        ("kv_heads", C.c_int32),
        ("max_q", C.c_int32),
        ("max_kv", C.c_int32),
        ("head_dim", C.c_int32),
        ("page_size", C.c_int32),
        ("is_causal", C.c_int32),
        ("device", C.c_int32),
        ("sm_scale", C.c_float),
    ]


class DecodeArgs(C.Structure):
    _fields_ = [
        ("q", C.c_void_p),
        ("k", C.c_void_p),
        ("v", C.c_void_p),
        ("out", C.c_void_p),
        ("kv_indptr", C.c_void_p),
        ("k_table", C.c_void_p),
        ("v_table", C.c_void_p),
        ("workspace", C.c_void_p),
        ("workspace_bytes", C.c_size_t),
        ("total_kv", C.c_int64),
        ("table_stride", C.c_int64),
        ("dtype", C.c_int32),
        ("layout", C.c_int32),
        ("indptr_is_i64", C.c_int32),
        ("batch", C.c_int32),
        ("q_heads", C.c_int32),
        ("kv_heads", C.c_int32),
        ("q_len", C.c_int32),
        ("max_kv", C.c_int32),
        ("head_dim", C.c_int32),
        ("page_size", C.c_int32),
        ("causal_drafts", C.c_int32),
        ("device", C.c_int32),
        ("sm_scale", C.c_float),
    ]


class PagedAppendArgs(C.Structure):
    _fields_ = [
        ("src", C.c_void_p),
        ("cache", C.c_void_p),
        ("src_indptr", C.c_void_p),
        ("dst_pos", C.c_void_p),
        ("table", C.c_void_p),
        ("workspace", C.c_void_p),
        ("workspace_bytes", C.c_size_t),
        ("total_rows", C.c_int64),
        ("cache_rows", C.c_int64),
        ("table_stride", C.c_int64),
        ("row_bytes", C.c_int32),
        ("indptr_is_i64", C.c_int32),
        ("batch", C.c_int32),
        ("page_size", C.c_int32),
        ("device", C.c_int32),
    ]


class SoftmaxArgs(C.Structure):
    _fields_ = [
        ("x", C.c_void_p),
        ("out", C.c_void_p),
        ("rows", C.c_int64),
        ("cols", C.c_int64),
        ("dtype", C.c_int32),
        ("log_softmax", C.c_int32),
        ("device", C.c_int32),
    ]


_lib: Optional[C.CDLL] = None
_lib_lock = threading.Lock()


def library_path() -> str:
    return os.environ.get("B200ATTN_LIBRARY", os.path.join(_PKG_ROOT, _LIB_NAME))


def lib() -> C.CDLL:
    """Load the shared object once; raise loudly if it is not there."""
    global _lib
    if _lib is not None:
        return _lib
    with _lib_lock:
        if _lib is not None:
            return _lib
        path = library_path()
        if not os.path.exists(path):
            raise RuntimeError(
                f"{_LIB_NAME} not found at {path}. Build it with `make -C {os.path.join(_PKG_ROOT, 'csrc')}` "
                "(needs nvcc with sm_100a support). There is no CPU or Triton fallback."
            )
        handle = C.CDLL(path)
        handle.b200attn_abi_version.restype = C.c_int
        handle.b200attn_last_error.restype = C.c_char_p
        handle.b200attn_device_info.argtypes = [C.c_int, C.POINTER(DeviceInfo)]
        handle.b200attn_device_info.restype = C.c_int
        handle.b200attn_prefill_workspace_bytes.argtypes = [C.POINTER(PrefillArgs)]
        handle.b200attn_prefill_workspace_bytes.restype = C.c_size_t
        handle.b200attn_decode_workspace_bytes.argtypes = [C.POINTER(DecodeArgs)]
        handle.b200attn_decode_workspace_bytes.restype = C.c_size_t
        handle.b200attn_decode_route.argtypes = [C.POINTER(DecodeArgs), C.c_int, C.c_int]
        handle.b200attn_decode_route.restype = C.c_int
        handle.b200attn_decode_keys_as_rows.argtypes = [C.POINTER(DecodeArgs), C.c_int, C.c_int]
        handle.b200attn_decode_keys_as_rows.restype = C.c_int
        handle.b200attn_prefill_route.argtypes = [C.POINTER(PrefillArgs), C.c_int]
        handle.b200attn_prefill_route.restype = C.c_int
        handle.b200attn_prefill.argtypes = [C.POINTER(PrefillArgs), C.c_void_p]
        handle.b200attn_prefill.restype = C.c_int
        handle.b200attn_decode.argtypes = [C.POINTER(DecodeArgs), C.c_void_p]
        handle.b200attn_decode.restype = C.c_int
        handle.b200attn_decode_static.argtypes = [C.POINTER(DecodeArgs), C.c_void_p]
        handle.b200attn_decode_static.restype = C.c_int
        handle.b200attn_decode_static_check.argtypes = [C.c_int, C.c_void_p, C.POINTER(C.c_int32)]
        handle.b200attn_decode_static_check.restype = C.c_int
        handle.b200attn_selftest_wait_expiry.argtypes = [C.c_int, C.c_void_p, C.c_uint32, C.c_void_p]
        handle.b200attn_selftest_wait_expiry.restype = C.c_int
        handle.b200attn_selftest_cluster_expiry.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_uint32, C.c_int, C.c_void_p]
        handle.b200attn_selftest_cluster_expiry.restype = C.c_int
        handle.b200attn_selftest_abandoned_units.argtypes = [C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_void_p]
        handle.b200attn_selftest_abandoned_units.restype = C.c_int
        handle.b200attn_paged_append.argtypes = [C.POINTER(PagedAppendArgs), C.c_void_p]
        handle.b200attn_paged_append.restype = C.c_int
        handle.b200attn_softmax.argtypes = [C.POINTER(SoftmaxArgs), C.c_void_p]
        handle.b200attn_softmax.restype = C.c_int
        handle.b200attn_check_workspace.argtypes = [C.c_void_p, C.c_void_p, C.POINTER(C.c_int32)]
        handle.b200attn_check_workspace.restype = C.c_int
        got = handle.b200attn_abi_version()
        if got != ABI_VERSION:
            raise RuntimeError(f"{path}: ABI version {got}, expected {ABI_VERSION}")
        _lib = handle
        return _lib


# ---------------------------------------------------------------------------
# The native call path (csrc/host.cpp).  ``fast`` is bound to the library at its first use; until then, and for calls
# it does not take (it answers None), the entry points validate and launch from Python.  It saves the caller's time and
# nothing else: where the extension is missing, or was built for another interpreter or torch, every call goes that way.
# ---------------------------------------------------------------------------
def _unbound(*_args):
    """Stands in for the functions of ``_host`` until the first call with CUDA tensors binds them."""
    if torch.cuda.is_available():
        bind_host()
    return None


class _Unbound:
    prefill = decode = paged_append = softmax = staticmethod(_unbound)

    @staticmethod
    def forget() -> None:
        pass


class _Python(_Unbound):
    """Takes no call: there is no ``_host`` to bind."""

    prefill = decode = paged_append = softmax = staticmethod(lambda *_args: None)


fast = _Unbound


def bind_host() -> None:
    """Load ``_host`` and hand it the library and the workspace table."""
    global fast
    lib()
    try:
        from . import _host
    except ImportError as e:
        warnings.warn(f"the native call path is not there ({e}): every call is validated and launched from Python, some 10 us "
                      f"slower. Build it with `make -C {os.path.join(_PKG_ROOT, 'csrc')}`.", RuntimeWarning, stacklevel=4)
        fast = _Python
        return
    _host.bind(library_path(), _host_workspace)
    fast = _host


def last_error() -> str:
    msg = lib().b200attn_last_error()
    return msg.decode("utf-8", "replace") if msg else ""


def check(status: int, what: str) -> None:
    if status != 0:
        raise RuntimeError(f"{what} failed with status {status}: {last_error()}")


def device_info(device: int) -> DeviceInfo:
    info = DeviceInfo()
    check(lib().b200attn_device_info(int(device), C.byref(info)), "b200attn_device_info")
    return info


# ---------------------------------------------------------------------------
# Workspace: one zero-initialised byte buffer per (device, stream), grown on demand.
# Word 0 is the device error code; kernels of the same stream reuse the rest.
# ---------------------------------------------------------------------------
HEADER_BYTES = 256  # error word, scheduling counters and merge tickets: zero before every call (include/b200attn.h)
_workspaces: Dict[Tuple[int, int], torch.Tensor] = {}
# buffers replaced by a larger one: a kernel still running may yet set its error word in one of them, so they are
# kept (alive and un-reused) until the next error check has read them
_retired: Dict[Tuple[int, int], list] = {}
# workspaces of calls that were recorded into a CUDA graph by a stream without one of its own (see _recorded_workspace)
_recorded: Dict[Tuple[int, int], torch.Tensor] = {}


def _capturing(device: torch.device) -> bool:
    with torch.cuda.device(device):
        return torch.cuda.is_current_stream_capturing()


def _recorded_workspace(key: Tuple[int, int], device: torch.device, nbytes: int) -> torch.Tensor:
    """Memory that is allocated while a stream records belongs to the graph's pool, where a replay of any graph of that pool
    may write over it, and a zero fill of it runs with that graph's replays, not now and not with another graph's.  So calls
    outside a capture never see this buffer, and every recorded call zeroes the counters and tickets itself."""
    buf = _recorded.get(key)
    if buf is None or buf.numel() < nbytes:
        if buf is not None:
            _retired.setdefault(key, []).append(buf)
        buf = _recorded[key] = torch.zeros((max(int(nbytes), 1 << 20) + 255) & ~255, dtype=torch.uint8, device=device)
    else:
        buf[4:HEADER_BYTES].zero_()  # (not the error word: nothing but check_device_errors clears that)
    return buf


def workspace(device: torch.device, stream_ptr: int, nbytes: int) -> torch.Tensor:
    key = (device.index if device.index is not None else torch.cuda.current_device(), int(stream_ptr))
    buf = _workspaces.get(key)
    if buf is None or buf.numel() < nbytes:
        if _capturing(device):
            return _recorded_workspace(key, device, nbytes)
        size = max(int(nbytes), 1 << 20)
        size = (size + 255) & ~255
        if buf is not None:
            _retired.setdefault(key, []).append(buf)
            fast.forget()  # its view of the table would keep pointing at the retired buffer
        buf = torch.zeros(size, dtype=torch.uint8, device=device)
        _workspaces[key] = buf
    return buf


def _host_workspace(device: torch.device, stream_ptr: int, nbytes: int) -> Tuple[torch.Tensor, bool]:
    """``workspace`` for the native call path, and whether the calls that follow on the stream may use it, too."""
    buf = workspace(device, stream_ptr, nbytes)
    return buf, any(buf is b for b in _workspaces.values())


def check_device_errors() -> None:
    """Synchronise and raise if any kernel launched so far recorded a device-side error
    (bounded wait expired, block-table entry out of range, planner overflow)."""
    code = C.c_int32(0)
    first_error = None
    for (dev, stream_ptr), buf in [*_workspaces.items(), *_recorded.items()]:
        for b in [buf] + _retired.pop((dev, stream_ptr), []):
            status = lib().b200attn_check_workspace(C.c_void_p(b.data_ptr()), C.c_void_p(stream_ptr), C.byref(code))
            if b is _recorded.get((dev, stream_ptr)) and code.value not in (1, 2, 3):
                continue  # not an error code: another graph of the pool wrote there
            if status != 0 and first_error is None:
                first_error = (status, f"device error check on cuda:{dev}", last_error())
    if first_error is not None:
        raise RuntimeError(f"{first_error[1]} failed with status {first_error[0]}: {first_error[2]}")


def release_workspaces() -> None:
    fast.forget()
    _workspaces.clear()
    _recorded.clear()
    _retired.clear()
