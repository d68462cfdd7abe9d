"""Loader of the in-tree native extension and the per-process kernel status word.

The extension is a plain pybind11 module (``meshslice_b200/_C*.so``) built by
``meshslice_b200.build``.  On a machine with a GPU a missing extension is an error: no op of
this package silently falls back to another implementation of a CUDA path.
"""
from __future__ import annotations

import importlib.util
import threading

_lock = threading.Lock()
_mod = None
_status = None
_cuda = None          # torch._C once CUDA is initialised

STATUS_NAMES = {
    0: "ok", 1: "timeout: producer waiting for a free stage", 2: "timeout: MMA waiting for TMA data",
    3: "timeout: MMA waiting for the epilogue", 4: "timeout: epilogue waiting for the accumulator",
    5: "timeout: waiting for a gathered chunk", 6: "timeout: bulk copy of the communication warp",
    7: "timeout: entry barrier with peers", 8: "timeout: exit barrier with peers",
    9: "timeout: reduce phase waiting for peers' partial tiles", 10: "timeout: waiting for the local go flag",
}


class KernelStatusError(RuntimeError):
    """A kernel of this package gave up on a bounded wait and reported an error code."""


def load():
    """Import (building if necessary and possible) and return the native module."""
    global _mod
    if _mod is not None:
        return _mod
    with _lock:
        if _mod is not None:
            return _mod
        from .build import ext_path
        path = ext_path()
        if not path.exists():
            from .build import build
            build()
        spec = importlib.util.spec_from_file_location("meshslice_b200._C", path)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        _mod = mod
    return _mod


def available() -> bool:
    try:
        load()
        return True
    except Exception:
        return False


def stream_ptr() -> int:
    """Current stream of the current device (asked for before every launch: without the stream object that
    torch.cuda.current_stream() builds, 0.2 us instead of 8)."""
    if _cuda is None:
        _init_cuda()
    return _cuda._cuda_getCurrentRawStream(_cuda._cuda_getDevice())


def _init_cuda():
    global _cuda
    import torch
    if not torch.cuda.is_initialized():
        torch.cuda.init()
    _cuda = torch._C


def _block_here(t) -> bool:
    """One block of memory on the current GPU, whose current stream a clear may go to."""
    if not (t.is_cuda and t.is_contiguous()):
        return False
    if _cuda is None:
        _init_cuda()
    return t.get_device() == _cuda._cuda_getDevice()


def zero_(t) -> None:
    """``t.zero_()`` without the tensor library's dispatch where the memory is one block on the current GPU."""
    if _block_here(t):
        load().memset_zero(t.data_ptr(), t.numel() * t.element_size(), stream_ptr())
    else:
        t.zero_()


def zero_both_(a, b) -> None:
    """``zero_`` of two tensors, in one launch where ``b`` follows ``a`` without a gap in the same block of the current GPU's memory."""
    n = a.numel() * a.element_size()
    if (_block_here(a) and _block_here(b) and b.data_ptr() == a.data_ptr() + n
            and a.untyped_storage().data_ptr() == b.untyped_storage().data_ptr()):
        load().memset_zero(a.data_ptr(), n + b.numel() * b.element_size(), stream_ptr())
    else:
        zero_(a)
        zero_(b)


class _Status:
    def __init__(self):
        C = load()
        self.host, self.dev = C.status_alloc()

    def read(self):
        return load().status_read(self.host)

    def clear(self):
        load().status_clear(self.host)


def status() -> _Status:
    """Host-mapped status word that every kernel launch of this process reports into."""
    global _status
    if _status is None:
        _status = _Status()
    return _status


def check_status(sync: bool = True) -> None:
    """Raise KernelStatusError if any kernel since the last check reported a timeout."""
    import torch
    if sync:
        torch.cuda.synchronize()
    st = status()
    code, blk, d0, d1 = st.read()
    if code != 0:
        st.clear()
        raise KernelStatusError(
            f"kernel status {code} ({STATUS_NAMES.get(code, '?')}), block {blk}, detail {d0}, {d1}")
