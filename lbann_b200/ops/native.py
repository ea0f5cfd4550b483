"""ctypes binding of the in-tree native libraries.

``cuda_lib()`` returns the sm_100a kernel library (``_native/liblbann_b200.so``) and
fails loudly when it is missing, so a GPU run never falls back to PyTorch kernels
silently.  ``host_lib()`` returns the C++ host runtime (checkpoint container, I/O
thread pool, graph utilities), which also works on CPU-only machines.
"""
from __future__ import annotations

import contextlib
import ctypes
import gc
import os
import threading

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
_NATIVE = os.path.join(os.path.dirname(_HERE), "_native")
_lock = threading.Lock()
_cuda = None
_host = None
_nodes = None

c_void_p = ctypes.c_void_p
c_int = ctypes.c_int
c_ll = ctypes.c_longlong
c_float = ctypes.c_float

DT_F16, DT_BF16, DT_F32 = 0, 1, 2
ACT_NONE, ACT_RELU, ACT_LEAKY, ACT_GELU, ACT_TANH, ACT_SIGMOID = 0, 1, 2, 3, 4, 5

STATUS_TEXT = {
    0: "ok",
    1: "timeout waiting for a TMA stage",
    2: "timeout waiting for a free pipeline stage",
    3: "timeout waiting for an accumulator",
    4: "timeout waiting for the epilogue to drain an accumulator",
    5: "timeout waiting for a flag from another rank",
    6: "bad argument seen on the device",
}


class NativeError(RuntimeError):
    pass


def dtype_code(dt: torch.dtype) -> int:
    if dt == torch.float16:
        return DT_F16
    if dt == torch.bfloat16:
        return DT_BF16
    if dt == torch.float32:
        return DT_F32
    raise NativeError(f"unsupported dtype {dt}")


def _load(name: str):
    path = os.path.join(_NATIVE, name)
    if not os.path.exists(path):
        # Build on demand (needs nvcc / g++); a GPU box normally receives the built files.
        from .. import _build
        _build.build_native()
    if not os.path.exists(path):
        raise NativeError(f"native library {path} is missing; run `python -m lbann_b200._build`")
    return ctypes.CDLL(path, mode=ctypes.RTLD_GLOBAL)


def cuda_lib():
    global _cuda
    if _cuda is None:
        with _lock:
            if _cuda is None:
                lib = _load("liblbann_b200.so")
                lib.lb_consume_status.restype = c_int
                lib.lb_consume_status.argtypes = [c_void_p]
                lib.lb_status_ptr.restype = c_void_p
                lib.lb_sm_count.restype = c_int
                lib.lb_stream_create.restype = c_int
                lib.lb_stream_create.argtypes = [ctypes.POINTER(c_void_p)]
                _cuda = lib
    return _cuda


_idle_streams = {}       # by device; as many as there were captures at the same time


@contextlib.contextmanager
def capture(graph, device, pool=None, empty_cache=False):
    """``with capture(graph, device)`` records into a ``torch.cuda.CUDAGraph``.  ``torch.cuda.graph`` always waits for
    the GPU and gives every cached block of the allocator back, which the next steps of all models allocate again:
    ``empty_cache``, for steps that need the memory.  Nor is its stream anybody's own: PyTorch hands 32 streams out
    again and again, and pinned memory that is freed meanwhile has an event recorded on each stream that read it, in
    whatever that stream is capturing."""
    key = torch.device(device).index or 0
    current = torch.cuda.current_stream(device)
    with _lock:
        idle = _idle_streams.setdefault(key, [])
        stream = idle.pop() if idle else None
    if stream is None:
        handle = c_void_p()
        with torch.cuda.device(key):
            check(cuda_lib().lb_stream_create(ctypes.byref(handle)), "lb_stream_create")
        stream = torch.cuda.ExternalStream(handle.value, device=key)
    if empty_cache:
        torch.cuda.synchronize(device)
        torch.cuda.empty_cache()
    stream.wait_stream(current)
    collecting = gc.isenabled()
    gc.disable()              # what a collection frees may not be allowed in a capture
    try:
        with torch.cuda.stream(stream):
            graph.capture_begin(*(() if pool is None else (pool,)), capture_error_mode="thread_local")
            try:
                yield
            finally:
                graph.capture_end()
    finally:
        if collecting:
            gc.enable()
    current.wait_stream(stream)
    with _lock:
        idle.append(stream)


def host_lib():
    global _host
    if _host is None:
        with _lock:
            if _host is None:
                _host = _load("liblbann_b200_host.so")
    return _host


def _load_nodes(lib, path: str):
    """The extension module at ``path``; NativeError unless it was built for the launchers of ``lib``
    (its calls bind to whatever library is loaded)."""
    import importlib.util
    if not os.path.exists(path):
        raise NativeError(f"native library {path} is missing; run `python -m lbann_b200._build`")
    spec = importlib.util.spec_from_file_location("_lbann_autograd", path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    built = getattr(mod, "abi_version", None)
    if built != lib.lb_abi_version():
        raise NativeError(f"{path} was built for version {built} of the launchers, the kernel library has "
                          f"{lib.lb_abi_version()}; run `python -m lbann_b200._build` and start again")
    mod.set_error_type(NativeError)
    return mod


def nodes():
    """The C++ autograd nodes (``csrc/autograd_nodes.cpp``): the launches of the tensor-core
    kernels and the forward / backward functions of the layers built on them."""
    global _nodes
    if _nodes is None:
        path = os.path.join(_NATIVE, "_lbann_autograd.so")
        if not os.path.exists(path):
            # before the kernel library is loaded, where that has not happened: the build may renew it
            from .. import _build
            _build.build_native()
        lib = cuda_lib()
        with _lock:
            if _nodes is None:
                _nodes = _load_nodes(lib, path)
    return _nodes


def have_cuda_lib() -> bool:
    return os.path.exists(os.path.join(_NATIVE, "liblbann_b200.so"))


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def stream_ptr() -> int:
    """The current CUDA stream's handle (the raw getter avoids building a Stream object on
    every kernel launch: ~17 us -> <1 us)."""
    if _raw_stream is not None:
        return _raw_stream(torch.cuda.current_device())
    return torch.cuda.current_stream().cuda_stream


def ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


def check(rc: int, what: str) -> None:
    if rc != 0:
        raise NativeError(f"{what} failed with code {rc}")


_status_listeners = []


def on_status(fn) -> None:
    """``fn(code)`` is called whenever ``consume_status`` finds a non-zero device status."""
    _status_listeners.append(fn)


def set_wait_budget_ns(ns: int) -> None:
    """Budget of the device-side waits on other ranks (0 restores the built-in 2 s)."""
    lib = cuda_lib()
    lib.lb_set_wait_budget_ns.restype = c_int
    lib.lb_set_wait_budget_ns.argtypes = [ctypes.c_ulonglong]
    check(lib.lb_set_wait_budget_ns(int(ns)), "lb_set_wait_budget_ns")


def consume_status(raise_on_error: bool = True) -> int:
    """Synchronise the current stream and return (and clear) the device status word."""
    code = cuda_lib().lb_consume_status(stream_ptr())
    if code:
        for fn in list(_status_listeners):
            fn(code)
    if code and raise_on_error:
        raise NativeError(f"device reported: {STATUS_TEXT.get(code, code)}")
    return code


_launch_count = 0


def count_launch(n: int = 1) -> None:
    """Bookkeeping for benchmarks: number of this library's kernels launched."""
    global _launch_count
    _launch_count += n


def launches() -> int:
    return _launch_count + (_nodes.launches() if _nodes is not None else 0)


def __getattr__(name):
    # how many launches were lent scratch for a split of their reduction (tests read it)
    if name == "splitk_offers":
        return _nodes.splitk_offers() if _nodes is not None else 0
    raise AttributeError(f"module '{__name__}' has no attribute '{name}'")
