"""ctypes binding of ``lib/libcpb.so`` (the sm_100a kernels and the C++ runtime).

The library has a plain C ABI: every launcher takes raw device pointers, sizes and a CUDA stream
and returns 0 or a negative error code whose text is available from ``cpb_last_error``.  Python
passes ``tensor.data_ptr()`` and the stream as plain integers; :func:`lib` declares every argument's type.

On a machine with a GPU a missing or unloadable library is a hard error: the CUDA ops never fall
back to PyTorch silently.
"""
from __future__ import annotations

import ctypes
import os
import threading
from ctypes import c_char_p, c_double, c_float, c_int, c_long, c_size_t, c_void_p
from pathlib import Path
from typing import Optional

import torch

_LIB: Optional[ctypes.CDLL] = None
_LOAD_LOCK = threading.Lock()
_CTYPES = {"p": c_void_p, "i": c_int, "l": c_long, "f": c_float, "d": c_double, "z": c_size_t}
_LIB_PATH = Path(__file__).resolve().parent / "lib" / "libcpb.so"


class NativeError(RuntimeError):
    pass


def lib_path() -> Path:
    return _LIB_PATH


def available() -> bool:
    return _LIB_PATH.exists()


def _declare(handle) -> None:
    """Declare every launcher's argument types: launchers take plain Python numbers, converted by ctypes in C.  Without the
    declaration ctypes passes a Python integer as a C ``int``, which cuts a device pointer to 32 bits."""
    try:
        handle.cpb_signatures.restype = c_char_p
    except AttributeError:
        raise NativeError(f"{_LIB_PATH} was built from other sources (it lacks cpb_signatures); "
                          "rebuild it: `python -m context_parallelism_b200._build`") from None
    for entry in handle.cpb_signatures().decode().split():
        name, codes = entry.split(":")
        getattr(handle, name).argtypes = [_CTYPES[c] for c in codes]
    handle.cpb_last_error.restype = c_char_p


def lib() -> ctypes.CDLL:
    """Load (once) and return the native library.  It is published only when every argument type is declared, so neither a
    failed load nor a second thread can get at a library whose launchers would take truncated pointers."""
    global _LIB
    if _LIB is None:
        with _LOAD_LOCK:
            if _LIB is None:
                if not _LIB_PATH.exists():
                    if os.environ.get("CPB_NO_AUTOBUILD", "0") == "1":
                        raise NativeError(f"{_LIB_PATH} is missing; run `python -m context_parallelism_b200._build`")
                    from . import _build
                    _build.build()
                # libnccl / libcudart are provided by the already-imported torch; load with global symbols visible
                handle = ctypes.CDLL(str(_LIB_PATH), mode=ctypes.RTLD_GLOBAL)
                _declare(handle)
                _LIB = handle
    return _LIB


def check(rc: int, what: str = "") -> None:
    if rc != 0:
        msg = lib().cpb_last_error().decode(errors="replace")
        raise NativeError(f"{what} failed (code {rc}): {msg}")


def stream_ptr(device=None) -> int:
    """The calling thread's current stream on ``device`` as an address (no ``torch.cuda.Stream`` object is made)."""
    idx = None if device is None else (device if isinstance(device, torch.device) else torch.device(device)).index
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if idx is None else idx)


def ptr(t: Optional[torch.Tensor]) -> int:
    return 0 if t is None else t.data_ptr()


LAUNCHES = [0]          # number of kernel launchers invoked (each launches exactly one of our kernels)
_FN_CACHE = {}
_PROFILE = None         # name -> list of (start event, end event) while a per-kernel device timing is being taken


def call(name: str, *args) -> None:
    """Invoke ``cpb_<name>`` (argument types as declared by its definition) and raise on error."""
    fn = _FN_CACHE.get(name)
    if fn is None:
        fn = getattr(lib(), "cpb_" + name)
        fn.restype = c_int
        _FN_CACHE[name] = fn
    LAUNCHES[0] += 1
    if _PROFILE is not None:
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        rc = fn(*args)
        e1.record()
        _PROFILE.setdefault(name, []).append((e0, e1))
    else:
        rc = fn(*args)
    if rc != 0:
        check(rc, name)


def profile_start() -> None:
    """Start timing every launcher call with a pair of CUDA events on the stream it is issued to (diagnostics:
    device time per kernel name without a profiler; for the cross-rank barrier kernels this is the time spent
    waiting for the slowest peer)."""
    global _PROFILE
    _PROFILE = {}


def profile_stop():
    """Stop timing; returns ``{name: (calls, total_ms)}`` after one device synchronisation."""
    global _PROFILE
    prof, _PROFILE = _PROFILE, None
    torch.cuda.synchronize()
    return {k: (len(v), sum(a.elapsed_time(b) for a, b in v)) for k, v in (prof or {}).items()}


# --------------------------------------------------------------------------- kernel status words
_STATUS_CODES = {1: "mbarrier wait timed out", 2: "peer/readiness flag wait timed out", 3: "index out of range"}


class KernelStatus:
    """A 4-int device word ``[code, site, block, aux]`` kernels report bounded-wait expiry and
    bounds-check failures into; the host turns a non-zero code into an exception."""

    def __init__(self, device):
        self.buf = torch.zeros(4, dtype=torch.int32, device=device)

    def ptr(self) -> int:
        return self.buf.data_ptr()

    def check(self, what: str = "kernel") -> None:
        code, site, block, aux = self.buf.tolist()
        if code != 0:
            self.buf.zero_()
            raise NativeError(f"{what}: {_STATUS_CODES.get(code, 'error %d' % code)} "
                              f"(site {site}, block {block}, aux {aux})")


_status_cache = {}


def status_for(device) -> KernelStatus:
    dev = device if isinstance(device, torch.device) else torch.device(device)
    key = dev.index if dev.index is not None else torch.cuda.current_device()
    st = _status_cache.get(key)
    if st is None:
        st = _status_cache[key] = KernelStatus(torch.device("cuda", key))
    return st


f, i, l = float, int, int
