"""Loads the compiled kernel library, declares its entry points, and calls them (through csrc/host/entry.cpp).

There is no fallback for the kernels: if the library cannot be built or loaded, or the device is not
sm_100, every call raises ``KernelError``.
"""
from __future__ import annotations

import ctypes
import threading

from ..errors import KernelError

_P = ctypes.c_void_p
_I = ctypes.c_int
_F = ctypes.c_float

# name -> argument types (every function returns int status)
_SIGNATURES = {
    "dl_gather_rows": [_P, _I, _I, _P, _P, _I, _I, _I, _I, _P],
    "dl_add_rmsnorm": [_P, _P, _I, _P, _P, _I, _I, _I, _F, _P],
    "dl_rope_cache_write": [_P, _I, _P, _I, _P, _I, _I, _P, _P, _I, _I, _P, _P, _P, _I, _P, _P, _I,
                            _I, _I, _I, _I, _I, _P, _P, _P, _I, _P],
    "dl_attention_generic": [_P, _I, _P, _I, _I, _P, _P, _I, _P, _P, _P, _I, _I, _I, _I, _I, _I, _F, _I, _F, _P, _P, _I, _I, _P, _P],
    "dl_swiglu": [_P, _P, _I, _P, _I, _I, _I, _P],
    "dl_gemm_f32": [_P, _I, _P, _P, _I, _I, _I, _I, _P],
    "dl_sample": [_P, _I, _I, _I, _P, _P, _P, _P, _P, _P, _I, _P],
    "dl_repetition_penalty": [_P, _I, _I, _I, _P, _I, _I, _P, _P, _P, _P, _P, _P, _P],
}

_lock = threading.Lock()
_lib = None
_checked_device = False
_entry = None                # the CPython module of csrc/host/entry.cpp
_callables = {}              # entry point -> its callable
_KINDS = {_P: "p", _I: "i", _F: "f", ctypes.c_long: "l", ctypes.c_longlong: "l"}


def declare(lib, signatures):
    for name, argtypes in signatures.items():
        try:
            fn = getattr(lib, name)
        except AttributeError as exc:
            raise KernelError(f"kernel library lacks entry point {name}") from exc
        fn.argtypes = argtypes
        fn.restype = ctypes.c_int


def library():
    """The loaded library (built on first use)."""
    global _lib
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is not None:
            return _lib
        from . import build
        path = build.build()
        try:
            lib = ctypes.CDLL(str(path))
        except OSError as exc:
            raise KernelError(f"cannot load {path}: {exc}") from exc
        declare(lib, _SIGNATURES)
        lib.dl_last_error.restype = ctypes.c_char_p
        lib.dl_last_error.argtypes = []
        lib.dl_device_arch.restype = ctypes.c_int
        lib.dl_sm_count.restype = ctypes.c_int
        lib.dl_set_dependent_launch.restype = ctypes.c_int
        lib.dl_set_dependent_launch.argtypes = [ctypes.c_int]
        # Library products (cuBLAS through torch, used for bfloat16 prompts of more than 128 rows) must
        # accumulate and reduce in float32 like the kernels here: no bfloat16 split-k reductions.
        import torch
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
        _lib = lib
        return lib


def register_signatures(signatures):
    """Entry points of kernels added later (each module declares its own)."""
    _SIGNATURES.update(signatures)
    if _lib is not None:
        declare(_lib, signatures)


class _CtypesEntry:
    """What csrc/host/entry.cpp does, by ctypes, for machines where it cannot be built: the same calls, about 2.5 us each dearer.  Sizes and
    strides are not read ahead (-1, None): the callers' own rules take over."""

    def kinds(self, handle, name):
        out = ctypes.create_string_buffer(65)
        fn = getattr(library(), name + "_kinds", None)
        return out.value.decode() if fn is not None and fn(out, 65) >= 0 else None

    def bind(self, handle, name):
        import torch
        fn, pointers = getattr(library(), name), [t is _P for t in _SIGNATURES[name]]

        def entry(*args):
            if len(args) != len(pointers):
                raise TypeError(f"the entry point takes {len(pointers)} arguments, got {len(args)}")
            try:
                return fn(*[a.data_ptr() if p and isinstance(a, torch.Tensor) else a for a, p in zip(args, pointers)])
            except ctypes.ArgumentError as exc:
                raise TypeError(str(exc)) from exc
        return entry

    def all_cuda(self, *tensors):
        return all(t is None or t.is_cuda for t in tensors)

    def row_stride(self, t):
        return -1

    def product(self, x, w):
        return None

    def empty(self, rows, width, half, like):
        import torch
        return torch.empty((rows, width), dtype=torch.bfloat16 if half else torch.float32, device=like.device)

    def stream(self):
        import torch
        return torch.cuda.current_stream().cuda_stream


def entry():
    """The module that calls the library's entry points (built on first use, like the library): tensors are passed as they are."""
    global _entry
    if _entry is None:
        import importlib.machinery
        import importlib.util
        from . import build
        lib = library()
        with _lock:
            if _entry is None:
                try:
                    path = str(build.build_entry())
                    loader = importlib.machinery.ExtensionFileLoader(build.ENTRY, path)
                    module = importlib.util.module_from_spec(importlib.util.spec_from_file_location(build.ENTRY, path, loader=loader))
                    loader.exec_module(module)
                except (KernelError, ImportError) as exc:
                    build._log(f"calls go through ctypes, a few microseconds each dearer outside captured steps: {str(exc).strip()}")
                    module = _CtypesEntry()
                module.handle = lib._handle
                _entry = module
    return _entry


def _bind(name):
    """The callable of an entry point, whose own kinds of arguments must be the declared ones."""
    module = entry()
    declared = "".join(_KINDS[t] for t in _SIGNATURES[name])
    found = module.kinds(module.handle, name)
    if found != declared:
        raise KernelError(f"{name}: the library's arguments ({found}) are not the declared ones ({declared})")
    _callables[name] = fn = module.bind(module.handle, name)
    return fn


def require_device():
    """Raise unless the current CUDA device can run the sm_100a kernels."""
    global _checked_device
    if _checked_device:
        return
    import torch
    if not torch.cuda.is_available():
        raise KernelError("no CUDA device: this library runs on NVIDIA B200 (sm_100) only "
                          "and has no CPU fallback")
    arch = library().dl_device_arch()
    if arch // 10 != 10:
        raise KernelError(f"the kernels are compiled for sm_100a; the current device reports "
                          f"compute capability {arch / 10:.1f}")
    _checked_device = True


def set_dependent_launch(on):
    """Switch programmatic dependent launch for later launches: kernels may begin, up to their
    first read of an earlier kernel's output, while that kernel is still finishing.  On unless
    the environment sets DOTLLM_DEPENDENT_LAUNCH=0; results are the same either way."""
    library().dl_set_dependent_launch(1 if on else 0)


def current_stream():
    """The current CUDA stream's handle, for a kernel launch.  ``torch.cuda.current_stream()`` builds
    a Python stream object after several device-index and environment look-ups, 10 - 15 us a call with
    a few hundred launches a step."""
    return (_entry or entry()).stream()


_empty_kinds = None


def empty(rows, width, dtype, like):
    """A contiguous [rows, width] tensor on ``like``'s device: ``torch.empty`` without its parsing of arguments for the two types that
    kernels write most."""
    global _empty_kinds
    if _empty_kinds is None:
        import torch
        _empty_kinds = {torch.float32: False, torch.bfloat16: True}
    half = _empty_kinds.get(dtype)
    if half is None or _entry is None:
        import torch
        return torch.empty((rows, width), dtype=dtype, device=like.device)
    return _entry.empty(rows, width, half, like)


def call(name, *args):
    """Call an entry point; pointers may be given as tensors (their first element), as addresses or as None."""
    fn = _callables.get(name)
    status = (fn or _bind(name))(*args)
    if status != 0:
        raise KernelError(f"{name}: {library().dl_last_error().decode(errors='replace')} (status {status})")


_sm_counts = {}


def sm_count():
    """Multiprocessors of the current device (0 without one)."""
    import torch
    device = torch._C._cuda_getDevice() if torch.cuda.is_initialized() else None
    if device not in _sm_counts:
        count = library().dl_sm_count()
        if device is None:
            return count
        _sm_counts[device] = count
    return _sm_counts[device]


_status = {}
_counters = []
_STATUS_TEXT = {1: "a producer's wait for a free shared-memory stage expired",
                2: "a block table named a page outside the pool",
                3: "a consumer's wait for a bulk copy expired",
                5: "an epilogue's wait for a product's sums or for its rows' factors expired",
                6: "a consumer's wait for room for a product's sums expired"}


def register_counters(tensor):
    """Arrival counters that kernels share between launches and leave zero.  A launch that gave up on
    a bounded wait may leave some of them counted; ``check_status`` clears them with the status word
    so that the launches after the error start from the state they expect."""
    _counters.append(tensor)


def status_word(device):
    """The per-device int32 that kernels with bounded waits set when a wait expires."""
    key = device.index
    if key not in _status:
        import torch
        _status[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status[key]


def check_status():
    """Raise if a kernel reported an expired wait since the last check (synchronises)."""
    for key, word in _status.items():
        code = int(word.item())
        if code:
            word.zero_()
            for counters in _counters:
                if counters.device.index == key:
                    counters.zero_()
            raise KernelError(f"a kernel on cuda:{key} gave up: {_STATUS_TEXT.get(code, code)}")
