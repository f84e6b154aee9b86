"""ctypes binding of libsbvr_b200.so (the C ABI declared in include/sbvr_b200.h).

There is no fallback: if the library is missing, importing this module raises; if a call
returns a non-zero status, a RuntimeError carrying `sbvr_strerror` is raised, as the reference
binding raised RuntimeError from `std::runtime_error` (reference sbvr/kernels/sbvr_kernel.cu:624-628).
"""
from __future__ import annotations

import ctypes
import functools
import importlib.util
import os
import threading

import torch  # noqa: F401  (the extension module resolves its symbols in torch's libraries)

_PKG_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB_PATH = os.path.join(_PKG_ROOT, "lib", "libsbvr_b200.so")

if not os.path.exists(LIB_PATH):
    raise ImportError(
        f"{LIB_PATH} not found: build it with `python sbvr-cpu-arm_b200/build.py` "
        "(there is no CPU or PyTorch fallback for the SBVR kernels)")

lib = ctypes.CDLL(LIB_PATH)

# The host path between the Python API and the library (csrc/pyext.cpp), an extension module beside it.
NATIVE_PATH = os.path.join(_PKG_ROOT, "lib", "_sbvr_native.so")
if not os.path.exists(NATIVE_PATH):
    raise ImportError(f"{NATIVE_PATH} not found: build it with `python sbvr-cpu-arm_b200/build.py`")
_spec = importlib.util.spec_from_file_location("_sbvr_native", NATIVE_PATH)
native = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(native)

_vp, _i, _sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
_ip = ctypes.POINTER(ctypes.c_int)

lib.sbvr_strerror.argtypes = [_i]
lib.sbvr_strerror.restype = ctypes.c_char_p
lib.sbvr_last_cuda_error.argtypes = []
lib.sbvr_last_cuda_error.restype = _i
lib.sbvr_last_timeout_where.argtypes = []
lib.sbvr_last_timeout_where.restype = ctypes.c_uint
lib.sbvr_last_timeout_info.argtypes = [_i]
lib.sbvr_last_timeout_info.restype = ctypes.c_uint
lib.sbvr_query.argtypes = [_i, _ip, _ip, _ip, _ip, _ip]
lib.sbvr_query.restype = _i
lib.sbvr_workspace_create.argtypes = [ctypes.POINTER(_vp), _i, _sz]
lib.sbvr_workspace_create.restype = _i
lib.sbvr_workspace_bytes.argtypes = [_i, _i, _i, _i, ctypes.POINTER(_sz)]
lib.sbvr_workspace_bytes.restype = _i
lib.sbvr_workspace_destroy.argtypes = [_vp]
lib.sbvr_workspace_destroy.restype = _i
lib.sbvr_workspace_status.argtypes = [_vp, _vp]
lib.sbvr_workspace_status.restype = _i
lib.sbvr_linear_folds.argtypes = [_i, _i, _i, _i, _i, _i, _i, ctypes.POINTER(_i)]
lib.sbvr_linear_folds.restype = _i
lib.sbvr_workspace_patience.argtypes = [_vp, ctypes.c_uint]
lib.sbvr_workspace_patience.restype = _i
lib.sbvr_decode_f16.argtypes = [_vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _i, _vp]
lib.sbvr_decode_f16.restype = _i
lib.sbvr_linear_f16.argtypes = [_vp, _vp, _vp, _i, _vp, _i, _vp, _vp, _i, _i, _i, _i, _i, _i, _vp, _vp]
lib.sbvr_linear_f16.restype = _i
lib.sbvr_linear_workspace_bytes.argtypes = [_i, _vp, _vp, _i, _vp, _i, _i, _i, _i, _i, _i, ctypes.POINTER(_sz)]
lib.sbvr_linear_workspace_bytes.restype = _i
lib.sbvr_linear_padded_f16.argtypes = [_vp, _i, _vp, _vp, _i, _vp, _i, _vp, _vp, _i, _i, _i, _i, _i, _i, _vp, _vp]
lib.sbvr_linear_padded_f16.restype = _i
lib.sbvr_linear_fused_f16.argtypes = [_i, _vp, _vp, _vp, _vp, ctypes.c_float, _vp, _vp, _i, _vp, _i, _vp, _vp, _i, _i, _i,
                                      _i, _i, _vp, _vp]
lib.sbvr_linear_fused_f16.restype = _i
lib.sbvr_popc_mm_f16.argtypes = [_vp, _vp, _i, _vp, _i, _i, _vp, _vp, _i, _vp, _i, _i, _vp, _vp, _i, _i, _i, _vp]
lib.sbvr_popc_mm_f16.restype = _i
lib.sbvr_linear_t_f16.argtypes = [_vp, _vp, _vp, _i, _vp, _i, _vp, _vp, _i, _i, _i, _i, _i, _vp, _vp]
lib.sbvr_linear_t_f16.restype = _i
lib.sbvr_encode_mse_f16.argtypes = [_vp, _i, _vp, _i, _i, _vp, _vp]
lib.sbvr_encode_mse_f16.restype = _i
lib.sbvr_encode_select_f16.argtypes = [_vp, _i, _vp, _vp, _i, _vp, _vp]
lib.sbvr_encode_select_f16.restype = _i
lib.sbvr_encode_pack.argtypes = [_vp, _i, _i, _i, _vp, _vp]
lib.sbvr_encode_pack.restype = _i
lib.sbvr_linear_f16_host.argtypes = [_vp, _vp, _vp, _i, _vp, _i, _vp, _vp, _i, _i, _i, _i, _i, _i, _vp, _vp]
lib.sbvr_linear_f16_host.restype = _i
lib.sbvr_linear_f16_noalloc.argtypes = [_vp, _vp, _vp, _i, _vp, _i, _vp, _vp, _i, _i, _i, _i, _i, _vp]
lib.sbvr_linear_f16_noalloc.restype = _i

_f = ctypes.c_float
lib.sbvr_add_rmsnorm_f16.argtypes = [_vp, _vp, _vp, _vp, _vp, _i, _i, _f, _vp]
lib.sbvr_add_rmsnorm_f16.restype = _i
lib.sbvr_rope_append_f16.argtypes = [_vp, _vp, _vp, _f, _vp, _vp, _i, _i, _i, _i, _i, _i, _vp]
lib.sbvr_rope_append_f16.restype = _i
lib.sbvr_attention_f16.argtypes = [_vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _f, _i, _vp]
lib.sbvr_attention_f16.restype = _i
lib.sbvr_rope_attention_f16.argtypes = [_vp, _vp, _vp, _f, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _f, _i, _vp]
lib.sbvr_rope_attention_f16.restype = _i
lib.sbvr_silu_mul_f16.argtypes = [_vp, _vp, _i, _i, _vp]
lib.sbvr_silu_mul_f16.restype = _i
lib.sbvr_embedding_f16.argtypes = [_vp, _vp, _vp, _i, _i, _vp]
lib.sbvr_embedding_f16.restype = _i
lib.sbvr_argmax_f16.argtypes = [_vp, _vp, _vp, _i, _i, _vp]
lib.sbvr_argmax_f16.restype = _i

lib.sbvr_allreduce_add_rmsnorm_f16.argtypes = [_vp, _vp, _vp, _i, _i, _i, _i, _sz, _vp, _vp, _vp, _vp, _i, _i, _f, _vp, _vp]
lib.sbvr_allreduce_add_rmsnorm_f16.restype = _i
lib.sbvr_linear_push_f16.argtypes = [_i, _vp, _vp, _vp, _vp, _f, _vp, _vp, _i, _vp, _i, _vp, _vp, _i, _i, _i, _i, _i, _vp, _vp]
lib.sbvr_linear_push_f16.restype = _i
lib.sbvr_ll_reduce_add_rmsnorm_f16.argtypes = [_vp, _vp, _i, _i, _i, _i, _vp, _vp, _vp, _vp, _i, _i, _f, _i, _vp, _vp]
lib.sbvr_ll_reduce_add_rmsnorm_f16.restype = _i
lib.sbvr_ll_reduce_add_rmsnorm_digits_f16.argtypes = [_vp, _vp, _i, _i, _i, _i, _vp, _vp, _vp, _vp, _i, _i, _f, _i, _i, _vp, _vp]
lib.sbvr_ll_reduce_add_rmsnorm_digits_f16.restype = _i
lib.sbvr_allreduce_add_rmsnorm_digits_f16.argtypes = [_vp, _vp, _vp, _i, _i, _i, _i, _sz, _vp, _vp, _vp, _vp, _i, _i, _f, _i, _vp, _vp]
lib.sbvr_allreduce_add_rmsnorm_digits_f16.restype = _i

EXPORTS = ["sbvr_linear_folds", "sbvr_linear_workspace_bytes", "sbvr_linear_padded_f16", "sbvr_encode_stats_f16", "sbvr_encode_advance", "sbvr_encode_run", "sbvr_popc_mm_f16", "sbvr_linear_t_f16", "sbvr_encode_mse_f16", "sbvr_encode_select_f16", "sbvr_encode_pack", "sbvr_rope_attention_f16", "sbvr_linear_fused_f16", "sbvr_allreduce_add_rmsnorm_f16", "sbvr_linear_push_f16", "sbvr_ll_reduce_add_rmsnorm_f16", "sbvr_ll_reduce_add_rmsnorm_digits_f16", "sbvr_allreduce_add_rmsnorm_digits_f16", "sbvr_add_rmsnorm_f16", "sbvr_rope_append_f16", "sbvr_attention_f16", "sbvr_silu_mul_f16",
           "sbvr_embedding_f16", "sbvr_argmax_f16", "sbvr_linear_f16_noalloc", "sbvr_workspace_bytes", "sbvr_strerror", "sbvr_last_cuda_error", "sbvr_last_timeout_where", "sbvr_last_timeout_info", "sbvr_query", "sbvr_workspace_create",
           "sbvr_workspace_destroy", "sbvr_workspace_status", "sbvr_workspace_patience", "sbvr_decode_f16", "sbvr_linear_f16",
           "sbvr_linear_f16_host"]


class EncodeResult(ctypes.Structure):
    """sbvr_encode_result_t of include/sbvr_b200.h."""
    _fields_ = [("group", _i), ("status", _i), ("mse", _f), ("cached_mse", _f), ("cached_at", _i),
                ("line", ctypes.c_ushort * 4), ("reserved", _i)]


class EncodeWalk(ctypes.Structure):
    """sbvr_encode_walk_t of include/sbvr_b200.h."""
    _fields_ = [("data", _vp), ("stats", _vp), ("lines", _vp), ("best_mse", _vp), ("best_at", _vp), ("scratch", _vp),
                ("result", _vp), ("unit", _vp * 2), ("bias", _vp * 2), ("R", _i * 2), ("B", _i * 2), ("per_dim", _i * 2),
                ("S", _i), ("groups", _i), ("s_search_num", _i), ("from_", _i), ("line0", _i), ("line1", _i), ("warm", _i),
                ("search", _i), ("misses", _i), ("append_at", _i), ("append", ctypes.c_ushort * 4), ("extend_ratio", ctypes.c_double), ("cutoff", ctypes.c_double)]


lib.sbvr_encode_stats_f16.argtypes = [_vp, _i, _vp, _vp]
lib.sbvr_encode_stats_f16.restype = _i
lib.sbvr_encode_advance.argtypes = [ctypes.POINTER(EncodeWalk), _vp]
lib.sbvr_encode_advance.restype = _i


class EncodeRecord(ctypes.Structure):
    """sbvr_encode_record_t of include/sbvr_b200.h."""
    _fields_ = [("group", _i), ("at", _i), ("mse", _f), ("line", ctypes.c_ushort * 4)]


class EncodeRun(ctypes.Structure):
    """sbvr_encode_run_t of include/sbvr_b200.h."""
    _fields_ = [("ctl", _vp), ("records", _vp), ("outcome", _vp), ("n", _i), ("capacity", _i), ("warmup", _i), ("window", _i),
                ("hist_n", _i), ("limit", _i), ("acceptable", ctypes.c_double), ("hist", ctypes.c_double * 64)]


ENCODE_DONE, ENCODE_LIMIT, ENCODE_FULL, ENCODE_CALLER, ENCODE_TIMEOUT = 1, 2, 3, 4, 5
lib.sbvr_encode_run.argtypes = [ctypes.POINTER(EncodeWalk), ctypes.POINTER(EncodeRun), _vp]
lib.sbvr_encode_run.restype = _i


class PushDesc(ctypes.Structure):
    """sbvr_push_desc_t of include/sbvr_b200.h."""
    _fields_ = [("peer_recv", ctypes.c_ulonglong * 16), ("step", ctypes.c_void_p), ("calls_per_step", ctypes.c_int),
                ("call_idx", ctypes.c_int), ("rank", ctypes.c_int), ("world", ctypes.c_int), ("rows_max", ctypes.c_int),
                ("reserved", ctypes.c_int)]


def strerror(rc: int) -> str:
    return lib.sbvr_strerror(rc).decode()


def check(rc: int, what: str = "sbvr") -> None:
    if rc != 0:
        extra = ""
        if rc == -4:
            extra = f" (cudaError {lib.sbvr_last_cuda_error()})"
        raise RuntimeError(f"{what}: {strerror(rc)}{extra}")


def query(device: int = 0) -> dict:
    vals = [ctypes.c_int(0) for _ in range(5)]
    check(lib.sbvr_query(device, *[ctypes.byref(v) for v in vals]), "sbvr_query")
    keys = ["sm_count", "smem_per_block_optin", "l2_bytes", "cc_major", "cc_minor"]
    return {k: v.value for k, v in zip(keys, vals)}


class Workspace:
    """Owns one `sbvr_workspace_t`: the device status word of the kernels' bounded waits, padded
    activations and partial sums of the batched kernel, staging buffers of the host-pointer call."""

    DEFAULT_BYTES = 32 << 20

    def __init__(self, device: int, nbytes: int = 0):
        self.handle = _vp()
        self.device = device
        self.nbytes = nbytes or self.DEFAULT_BYTES
        check(lib.sbvr_workspace_create(ctypes.byref(self.handle), device, nbytes), "sbvr_workspace_create")

    def status(self, stream: int) -> int:
        return lib.sbvr_workspace_status(self.handle, _vp(stream))

    def close(self):
        if self.handle:
            lib.sbvr_workspace_destroy(self.handle)
            self.handle = _vp()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


_workspaces: dict = {}
# Workspaces replaced by larger ones.  They are never freed: a captured CUDA graph keeps the raw pointers of the
# workspace its kernels were recorded with (status word, counters, scratch), and would write into freed memory
# on replay if the replaced allocation went back to the driver.
_retired: list = []
# Torch's threads share the default stream, and creating a workspace lets other threads run.
_ws_lock = threading.Lock()


@functools.lru_cache(maxsize=4096)
def linear_folds(device: int, M: int, N: int, K: int, S: int, G: int, idx_bytes: int) -> bool:
    out = _i(0)
    check(lib.sbvr_linear_folds(device, M, N, K, S, G, idx_bytes, ctypes.byref(out)), "sbvr_linear_folds")
    return bool(out.value)


def workspace_bytes(device: int, M: int, N: int, K: int) -> int:
    out = _sz(0)
    check(lib.sbvr_workspace_bytes(device, M, N, K, ctypes.byref(out)), "sbvr_workspace_bytes")
    return out.value


def workspace(device: int, stream: int, nbytes: int = 0) -> Workspace:
    """One workspace per (device, stream): calls on one stream are ordered, so they may share scratch.
    A workspace smaller than `nbytes` is replaced by a larger one; the old one stays allocated for the life of the
    process (graphs captured earlier on this stream, and calls of other threads, still point into it)."""
    key = (device, stream)
    ws = _workspaces.get(key)
    if ws is not None and ws.nbytes >= nbytes:
        return ws
    with _ws_lock:                                 # one thread creates, the others find what it made
        ws = _workspaces.get(key)
        if ws is None or ws.nbytes < nbytes:
            new = Workspace(device, max(nbytes, Workspace.DEFAULT_BYTES))
            if ws is not None:
                _retired.append(ws)
            native.set_workspace(device, stream, new.handle.value, new.nbytes)
            _workspaces[key] = ws = new
    return ws


native.set_workspace_callback(workspace)
