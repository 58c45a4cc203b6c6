"""ctypes binding of ``libtrakb200.so`` (the C ABI declared in ``include/trak_b200.h``).

There is no fallback: if the shared library is missing or a call fails, the
caller gets an exception.
"""
import ctypes
import os
import threading

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "libtrakb200.so")

TB_F16, TB_BF16, TB_F32 = 0, 1, 2
TB_RADEMACHER, TB_NORMAL = 0, 1
TB_OK = 0
TB_ERR_BAD_PROJ_DIM = 3
TB_ERR_DEVICE_TIMEOUT = 7
TB_ERR_NOT_SPD = 10

_lib = None
_lock = threading.Lock()

_i, _i64, _u32 = ctypes.c_int, ctypes.c_int64, ctypes.c_uint32
_vp, _sz, _f = ctypes.c_void_p, ctypes.c_size_t, ctypes.c_float
_i32 = ctypes.c_int32


class Segment(ctypes.Structure):
    """tb_segment: one parameter's per-sample gradients ([B, numel], rows row_stride apart)."""
    _fields_ = [("ptr", ctypes.c_void_p), ("numel", ctypes.c_int64), ("row_stride", ctypes.c_int64)]


# name -> (restype, argtypes); one entry per function include/trak_b200.h declares
SIGNATURES = {
    "tb_version": (_i, []),
    "tb_strerror": (ctypes.c_char_p, [_i]),
    "tb_last_cuda_error": (ctypes.c_char_p, []),
    "tb_device_status": (_i, [_i, ctypes.POINTER(_u32)]),
    "tb_stream_status": (_i, [_i, _vp, ctypes.POINTER(_u32)]),
    "tb_selftest_wait_timeout": (_i, [_i, _vp, _u32]),
    "tb_selftest_sqrt": (_i, [_i, _vp, ctypes.c_uint64, ctypes.c_uint64, _vp]),
    "tb_project_workspace_bytes": (_sz, [_i, _i64, _i64, _u32, _u32]),
    "tb_project_least_workspace_bytes": (_sz, [_i, _i64, _i64, _u32, _u32, _i32]),
    "tb_project_grid": (_i, [_i64, _i64, _u32, _u32, _i, _i, ctypes.POINTER(_u32)]),
    "tb_profile_events": (_i, [_vp, _vp]),
    "tb_project_segments_workspace_bytes": (_sz, [_i, _i64, _i64, _u32, _u32, _i32]),
    "tb_project_segments": (_i, [_i, _vp, ctypes.POINTER(Segment), _i32, _i, _i64, _vp, _i64, _u32, _u32, _u32,
                                 _i, _f, _i, _vp, _sz]),
    "tb_gram_workspace_bytes": (_sz, [_i, _i64, _i64]),
    "tb_gram": (_i, [_i, _vp, _vp, _i, _i64, _i64, _i64, _vp, _i64, _i, _vp, _sz]),
    "tb_spd_inverse_workspace_bytes": (_sz, [_i64]),
    "tb_spd_inverse": (_i, [_i, _vp, _vp, _i64, _i64, _f, _i, _vp, _vp, _sz]),
    "tb_gemm_nt_workspace_bytes": (_sz, [_i, _i64, _i64, _i64]),
    "tb_gemm_nt_pack": (_i, [_i, _vp, _vp, _i64, _i, _i64, _i64, _i64, _vp, _sz]),
    "tb_gemm_nt_pack_beside": (_i, [_i, _vp, _vp, _i64, _i, _i64, _i64, _i64, _vp, _sz]),
    "tb_gemm_nt_packed": (_i, [_i, _vp, _vp, _i64, _i, _i64, _i64, _i64, _vp, _i64, _vp, _f, _i, _vp, _sz]),
    "tb_gemm_nt": (_i, [_i, _vp, _vp, _i64, _vp, _i64, _i, _i64, _i64, _i64, _vp, _i64, _vp, _f, _i, _vp, _sz]),
    "tb_matrix_bytes": (_sz, [_i64, _u32, _u32]),
    "tb_matrix_generate": (_i, [_i, _vp, _i64, _u32, _u32, _u32, _i, _i, _vp, _sz]),
    "tb_project_cached": (_i, [_i, _vp, _vp, _i, _i64, _i64, _i64, _vp, _i64, _u32, _u32, _vp, _sz, _f, _i, _vp, _sz]),
    "tb_project_segments_cached": (_i, [_i, _vp, ctypes.POINTER(Segment), _i32, _i, _i64, _vp, _i64, _u32, _u32, _vp,
                                        _sz, _f, _i, _vp, _sz]),
    "tb_finalize_scores": (_i, [_i, _vp, _vp, _i64, _vp, _i64, _i64, _f, _vp, _i, _i64]),
    "tb_project_static": (_i, [_i, _vp, _vp, _i, _i64, _i64, _i64, _vp, _i64, _u32, _u32, _u32, _i, _f, _i]),
    "tb_host_to_device": (_i, [_i, _vp, _vp, _vp, _sz]),
    "tb_device_to_host": (_i, [_i, _vp, _vp, _vp, _sz, _i]),
    "tb_host_threads": (_i, [ctypes.POINTER(_i)]),
    "tb_host_staging_release": (_i, []),
    "tb_project": (_i, [_i, _vp, _vp, _i, _i64, _i64, _i64, _vp, _i64, _u32, _u32, _u32, _i, _f, _i,
                        _vp, _sz]),
}


def lib():
    """The loaded library.  Raises ImportError (with the build hint) when absent."""
    global _lib
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is None:
            if not os.path.exists(LIB_PATH):
                raise ImportError(
                    f"{LIB_PATH} not found: build it with `python -m trak_b200.build` "
                    "(needs nvcc; the kernels are sm_100a only and there is no CPU fallback)")
            l = ctypes.CDLL(LIB_PATH)
            for name, (res, args) in SIGNATURES.items():
                fn = getattr(l, name)
                fn.restype = res
                fn.argtypes = args
            _lib = l
    return _lib


class DeviceTimeout(RuntimeError):
    pass


class NotPositiveDefinite(RuntimeError):
    """tb_spd_inverse met a non-positive Cholesky pivot (torch.linalg.inv of the reference would
    return garbage or raise on such a matrix)."""


def check(rc: int) -> None:
    """Maps a status code to the exception type the reference raises for it:
    ValueError for a bad projection dimension (std::invalid_argument in
    fast_jl/fast_jl_kernel.cuh:113-115), RuntimeError otherwise."""
    if rc == TB_OK:
        return
    l = lib()
    msg = l.tb_strerror(rc).decode()
    if rc == TB_ERR_BAD_PROJ_DIM:
        raise ValueError(msg)
    if rc == 6:
        msg = f"CUDA error: {l.tb_last_cuda_error().decode()}"
    if rc == TB_ERR_DEVICE_TIMEOUT:
        raise DeviceTimeout(msg)
    if rc == TB_ERR_NOT_SPD:
        raise NotPositiveDefinite(msg)
    raise RuntimeError(f"trak_b200: {msg} (code {rc})")


def device_status(device: int) -> None:
    """Synchronises the device and raises DeviceTimeout if a kernel gave up a wait."""
    detail = _u32(0)
    rc = lib().tb_device_status(device, ctypes.byref(detail))
    if rc == TB_ERR_DEVICE_TIMEOUT:
        raise DeviceTimeout(f"trak_b200: a bounded wait inside a kernel ran out (status {detail.value})")
    check(rc)


def stream_status(device: int, stream: int) -> None:
    """Waits for the work queued on ``stream`` and raises what ``device_status`` would raise for it."""
    detail = _u32(0)
    rc = lib().tb_stream_status(device, stream, ctypes.byref(detail))
    if rc == TB_ERR_DEVICE_TIMEOUT:
        raise DeviceTimeout(f"trak_b200: a bounded wait inside a kernel ran out (status {detail.value})")
    check(rc)


def current_stream(device: torch.device) -> int:
    """The handle of torch's current stream on ``device``."""
    return torch._C._cuda_getCurrentRawStream(device.index)


class on_device:
    """``torch.cuda.device(device)`` that costs next to nothing where ``device`` is the current one already."""

    __slots__ = ("guard",)

    def __init__(self, device: torch.device):
        self.guard = None if torch.cuda.current_device() == device.index else torch.cuda.device(device)

    def __enter__(self):
        if self.guard is not None:
            self.guard.__enter__()

    def __exit__(self, *exc):
        if self.guard is not None:
            self.guard.__exit__(*exc)
        return False


class Workspaces:
    """Scratch buffers kept by device and stream.  A buffer is its taker's alone until everything that uses it has been
    queued and it is given back; the stream orders the next user behind that.  (Were it left in the cache meanwhile, two
    threads that queue work on one stream would write over each other's operands between their launches.)"""

    def __init__(self, most_kept: int = 8):   # per process; streams come and go, their buffers should not pile up
        self.most_kept, self.kept = most_kept, {}

    def take(self, device: torch.device, stream: int, nbytes: int, least=None) -> torch.Tensor:
        """A buffer of ``nbytes``; where the device has no room for that, of the smaller size that ``least``, a function
        and its arguments, gives."""
        ws = self.kept.pop((device.index, stream), None)
        if ws is not None and ws.numel() >= nbytes:
            return ws
        size = 0 if ws is None else ws.numel()
        smaller = nbytes if least is None else min(nbytes, least[0](*least[1:]))
        if smaller < nbytes:
            if self.room(device) + size < nbytes:
                nbytes = smaller
            else:
                ws, size = None, 0   # given up before its successor is allocated
                try:
                    return torch.empty(nbytes, dtype=torch.uint8, device=device)
                except torch.cuda.OutOfMemoryError:
                    nbytes = smaller
        if size < nbytes:
            ws = None
            ws = torch.empty(max(nbytes, 256), dtype=torch.uint8, device=device)
        return ws

    @staticmethod
    def room(device: torch.device) -> int:
        """Bytes that can be allocated, fragmentation apart (which ``take`` finds out by trying)."""
        if device.type != "cuda" or torch.cuda.is_current_stream_capturing():
            return 1 << 62
        return torch.cuda.mem_get_info(device)[0] + torch.cuda.memory_reserved(device) - torch.cuda.memory_allocated(device)

    def give(self, device: torch.device, stream: int, ws: torch.Tensor) -> None:
        self.kept[(device.index, stream)] = ws  # most recently used last
        while len(self.kept) > self.most_kept:
            self.kept.pop(next(iter(list(self.kept))), None)

    def clear(self) -> None:
        self.kept.clear()
