"""ctypes binding of the C ABI declared in include/pragnosia_b200.h.

There is no fallback: if the shared library is missing, or a call returns a non-zero status, a RuntimeError is raised.
"""
from __future__ import annotations

import contextlib
import ctypes as C
import gc
import importlib.util
import threading
from pathlib import Path

import torch

PKG = Path(__file__).resolve().parent
LIB_PATH = PKG / "lib" / "libpragnosia_b200.so"
HOST_PATH = PKG / "lib" / "pgb_torch.so"

F32, BF16 = 0, 1
PREFILL_AUTO, PREFILL_FP32, PREFILL_TENSOR = 0, 1, 2

_vp, _ll, _i, _f = C.c_void_p, C.c_longlong, C.c_int, C.c_float

# name -> argument types (every entry point returns int except the two string getters)
SIGNATURES = {
    "pgb_abi_version": [],
    "pgb_lambda_scan_fwd": [_vp, _vp, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _vp],
    "pgb_lambda_scan_fwd_ex": [_vp, _vp, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_aspin_prep_fwd": [_vp, _vp, _vp, _i, _ll, _ll, _ll, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _vp],
    "pgb_aspin_prefill_fwd": [_vp, _vp, _vp, _i, _vp, _vp, _vp, _vp, _vp, _f, _vp, _i, _vp, _vp, _i, _i, _i, _i, _i, _vp],
    "pgb_aspin_prefill_segments_scratch_bytes": [_i, _i, _i, _i],
    "pgb_aspin_prefill_segments_fwd": [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _f, _vp, _i, _vp, _vp, _vp, _ll, _i, _i, _i, _i, _vp],
    "pgb_aspin_prefill_train_fwd": [_vp] * 9 + [_ll, _i, _i, _i, _i, _vp],
    "pgb_aspin_prefill_fp32_scratch_bytes": [_i, _i, _i, _i],
    "pgb_aspin_prefill_fp32_fwd": [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _f, _vp, _i, _vp, _vp, _vp, _ll, _i, _i, _i, _i, _vp],
    "pgb_aspin_delta_prefill_fwd": [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _f, _vp, _i, _vp, _vp, _vp, _ll, _i, _i, _i, _i, _vp],
    "pgb_aspin_delta_scratch_bytes": [_i, _i, _i],
    "pgb_aspin_delta_prefill_scratch_bytes": [_i, _i, _i, _i],
    "pgb_aspin_delta_prefill_noscratch_fwd": [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _f, _vp, _i, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_aspin_delta_prefill_train_fwd": [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _ll, _i, _i, _i, _i, _vp],
    "pgb_aspin_train_scratch_bytes": [_i, _i, _i, _i, _i],
    "pgb_aspin_train_bwd": [_vp] * 18 + [_ll, _i, _i, _i, _i, _vp],
    "pgb_aspin_prefill_fused_fwd": [_vp, _vp, _vp, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _f, _vp, _f, _vp, _i, _vp, _vp,
                                    _i, _i, _i, _i, _vp],
    "pgb_aspin_layer_prefill_fwd": [_vp, _vp, _vp, _ll, _ll, _vp, _vp, _ll, _ll, _vp, _vp, _i, _vp, _vp, _vp, _f, _vp, _f,
                                    _vp, _i, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_aspin_layer_windows_scratch_bytes": [_i, _i, _i, _i],
    "pgb_aspin_layer_prefill_windows_fwd": [_vp, _vp, _vp, _ll, _ll, _vp, _vp, _ll, _ll, _vp, _vp, _i, _vp, _vp, _f, _vp, _vp, _vp, _ll,
                                            _i, _i, _i, _i, _i, _vp],
    "pgb_aspin_layer_prefill_windows_ex": [_vp, _vp, _vp, _ll, _ll, _vp, _vp, _ll, _ll, _vp, _vp, _i, _vp, _vp, _vp, _f, _vp, _vp, _vp, _ll,
                                           _i, _i, _i, _i, _i, _vp],
    "pgb_aspin_delta_layer_scratch_bytes": [_i, _i, _i, _i],
    "pgb_aspin_delta_layer_scratch_least_bytes": [_i, _i, _i, _i],
    "pgb_aspin_delta_layer_windows_fwd": [_vp, _vp, _vp, _ll, _ll, _vp, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _f, _vp, _vp, _vp, _ll,
                                          _i, _i, _i, _i, _i, _vp],
    "pgb_aspin_delta_layer_windows_ex": [_vp, _vp, _vp, _ll, _ll, _vp, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _vp, _f, _vp, _vp, _vp, _ll,
                                         _i, _i, _i, _i, _i, _vp],
    "pgb_rot_table_build": [_vp, _vp, _i, _i, _i, _vp],
    "pgb_add_norm": [_vp, _vp, _vp, _vp, _f, _i, _vp, _vp, _ll, _i, _i, _vp],
    "pgb_decode_embed": [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_decode_sample": [_vp, _i, _f, C.c_ulonglong, _vp, _vp, _i, _vp, _vp, _vp, _vp, _i, _i, _i, _vp],
    "pgb_decode_sample_ex": [_vp, _i, _f, _f, C.c_ulonglong, _vp, _vp, _i, _vp, _vp, _vp, _vp, _i, _i, _i, _vp],
    "pgb_batch_linear": [_vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_batch_linear_ex": [_vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp, _i, _vp, _vp, _i, _f, _vp, _vp, _i, _vp],
    "pgb_batch_linear_parts": [_i],
    "pgb_decode_embed_ex": [_vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_decode_embed_norm": [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_decode_linear_takes": [_i, _i, _i],
    "pgb_decode_linear_parts": [_i, _i, _i],
    "pgb_decode_linear_rounds": [_i, _i, _i, _i],
    "pgb_decode_linear": [_vp, _vp, _vp, _vp, _i, _f, _i, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_decode_advance": [_vp, _vp, _i, _vp],
    "pgb_decode_token_work_bytes": [_i, _i, _i, _i],
    "pgb_decode_token_wait_selftest": [_vp, _ll, _vp],
    "pgb_decode_token_fwd": [_vp, _i, _vp, _vp, _vp, _vp, _i, _f, _vp, _vp, _vp, _vp, _ll, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i,
                             _i, _vp],
    "pgb_decode_token_step_fwd": [_vp, _i, _vp, _vp, _vp, _vp, _i, _f, _vp, _vp, _vp, _i, _vp, _ll, _vp, _vp, _i, _i, _i, _i, _i, _i, _i,
                                  _i, _i, _vp],
    "pgb_decode_flow_wait_selftest": [_vp, _vp, _ll, _ll, _vp],
    "pgb_decode_flow_work_bytes": [_i, _i, _i, _i, _i],
    "pgb_decode_flow_step_fwd": [_vp, _i, _vp, _vp, _vp, _vp, _i, _f, _vp, _vp, _vp, _i, _vp, _ll, _vp, _vp, _i, _i, _i, _i, _i, _i, _i,
                                 _i, _i, _vp],
    "pgb_tc_wait_selftest": [_ll, _vp],
    "pgb_linear_act": [_vp, _vp, _vp, _vp, _ll, _i, _i, _i, _vp],
    "pgb_skinny_linear": [_vp, _vp, _vp, _vp, _i, _f, _vp, _vp, _i, _vp, _vp, _i, _i, _i, _vp],
    "pgb_tc_error_flag": [_vp],
    "pgb_tc_set_variant": [_i],
    "pgb_variants": [],
    "pgb_linear_act_set_variant": [_i],
    "pgb_decode_set_variant": [_i],
    "pgb_rotate_pairs": [_vp, _i, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_skinny_linear_ex": [_vp, _vp, _vp, _vp, _i, _f, _vp, _vp, _i, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_lambda_scan_time_segments": [_i, _i, _i, _i],
    "pgb_lambda_scan_fwd_train": [_vp, _vp, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _vp],
    "pgb_lambda_scan_bwd": [_vp, _vp, _vp, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _vp],
    "pgb_aspin_prep_bwd": [_vp, _vp, _vp, _i, _ll, _ll, _ll, _vp, _ll, _ll, _vp, _vp, _vp, _vp, _vp, _i, _vp, _vp, _vp, _vp, _vp,
                           _i, _i, _i, _i, _vp],
    "pgb_aspin_prep_bwd_tiles": [_i],
    "pgb_assoc_out_fwd": [_vp, _vp, _vp, _i, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_prefix_scan_fwd": [_vp, _vp, _i, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_assoc_out_bwd": [_vp, _vp, _vp, _i, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_prefix_scan_bwd": [_vp, _vp, _i, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_delta_inv_bwd": [_vp, _i, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_delta_loop_bwd": [_vp, _vp, _i, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_delta_inv_fwd": [_vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_delta_loop_fwd": [_vp, _vp, _i, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_key_topk_mask": [_vp, _i, _ll, _ll, _ll, _i, _i, _i, _i, _i, _vp],
    "pgb_short_conv_fwd": [_vp, _i, _ll, _ll, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp],
    "pgb_aspin_decode_step": [_vp, _vp, _vp, _i, _ll, _i, _vp, _ll, _i, _i, _vp, _ll, _vp, _vp, _vp, _f, _vp, _vp, _vp,
                              _f, _vp, _i, _ll, _i, _i, _i, _vp],
    "pgb_aspin_decode_step_ex": [_vp, _vp, _vp, _i, _ll, _i, _vp, _ll, _i, _i, _vp, _ll, _vp, _vp, _vp, _f, _vp, _vp, _vp,
                              _f, _vp, _i, _ll, _i, _i, _i, _i, _vp],
}

_lib = None


def lib() -> C.CDLL:
    """The loaded library; raises if it has not been built (python -m pragnosia_b200.build)."""
    global _lib
    if _lib is None:
        if not LIB_PATH.exists():
            raise RuntimeError(f"{LIB_PATH} is missing: build it with `python -m pragnosia_b200.build`. "
                               "pragnosia_b200 has no CPU or PyTorch fallback.")
        L = C.CDLL(str(LIB_PATH))
        for name, args in SIGNATURES.items():
            fn = getattr(L, name)
            fn.argtypes = args
            fn.restype = _ll if name.endswith("_bytes") else _i
        L.pgb_status_string.argtypes = [_i]; L.pgb_status_string.restype = C.c_char_p
        L.pgb_last_cuda_error.argtypes = []; L.pgb_last_cuda_error.restype = C.c_char_p
        _lib = L
    return _lib


_host = None


def host():
    """The C++ half of the tensor-level wrappers (csrc/torch_host.cpp): an extension module beside the library it calls."""
    global _host
    if _host is None:
        lib()
        if not HOST_PATH.exists():
            raise RuntimeError(f"{HOST_PATH} is missing: build it with `python -m pragnosia_b200.build`.")
        spec = importlib.util.spec_from_file_location(HOST_PATH.stem, HOST_PATH)
        _host = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(_host)
    return _host


def check(status: int, what: str) -> None:
    if status != 0:
        L = lib()
        msg = L.pgb_status_string(status).decode()
        extra = L.pgb_last_cuda_error().decode() if status == 6 else ""
        raise RuntimeError(f"{what}: {msg}" + (f" [{extra}]" if extra else ""))


def type_code(dt: torch.dtype) -> int:
    if dt is torch.float32:
        return F32
    if dt is torch.bfloat16:
        return BF16
    raise TypeError(f"pragnosia_b200 kernels take float32 or bfloat16 tensors, got {dt}")


def dtype_code(t: torch.Tensor) -> int:
    return type_code(t.dtype)


def ptr(t) -> int | None:
    return None if t is None else t.data_ptr()


_raw_stream = torch._C._cuda_getCurrentRawStream if hasattr(torch._C, "_cuda_getCurrentRawStream") else None


def stream_of(t: torch.Tensor) -> int:
    if _raw_stream is not None:                                       # no Stream object in between: a tenth of the time, per call
        return _raw_stream(t.get_device())
    return torch.cuda.current_stream(t.device).cuda_stream


_gpus = None


def one_gpu() -> bool:
    """True once CUDA is up and shows a single GPU: there is then no other device to switch to."""
    global _gpus
    if _gpus is None and torch.cuda.is_initialized():
        _gpus = torch.cuda.device_count()
    return _gpus == 1


def sm_count(device) -> int:
    return torch.cuda.get_device_properties(device).multi_processor_count


def on_device_of(fn):
    """Decorator for the tensor-level wrappers: the library reads CUDA's CURRENT device (SM count, kernel attributes, its
    per-device scratch array and error flags), so a call whose first tensor lives on another GPU runs with that GPU made
    current for its duration. Same device (the usual case): no context switch, no cost."""
    import functools

    @functools.wraps(fn)
    def run(*args, **kw):
        if one_gpu() or torch.compiler.is_compiling():
            return fn(*args, **kw)
        for a in args:
            if isinstance(a, torch.Tensor):
                if a.is_cuda and a.get_device() != torch.cuda.current_device():
                    with torch.cuda.device(a.device):
                        return fn(*args, **kw)
                break
        return fn(*args, **kw)
    return run


def need_cuda(*ts) -> None:
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("pragnosia_b200 ops run on CUDA tensors only (there is no CPU path)")


_capture_lock = threading.RLock()


class _Mark:
    """Where a stream stands behind the last constants made on it. Recorded once per call (mark_constants) or, failing that, by the first
    other stream that wants them: an event after every one of them cost a model's first pass 0.3 ms of 4.5."""
    __slots__ = ("event", "stream", "due")

    def __init__(self, device):
        self.event, self.stream, self.due = torch.cuda.Event(), torch.cuda.current_stream(device), False

    def record(self):
        self.event.record(self.stream)
        self.due = False


_marks = {}                                                       # (device, raw stream) -> _Mark


def mark_constants(t: torch.Tensor) -> None:
    """Mark what the calls so far have cached on the current stream (of t's device), if anything is new."""
    mark = _marks.get((t.get_device(), stream_of(t)))
    if mark is not None and mark.due and not torch.cuda.is_current_stream_capturing():
        mark.record()


class Cached:
    """Tensors that one call made for all the later ones. Another stream than the one they were made on waits for the kernels that
    made them, and the allocator is told, so that a cache replaced meanwhile is not handed out under that stream's kernels. A copy
    of the module that holds one starts without it. What is made while the caller's stream is captured has no contents until that
    graph is replayed: keep() leaves it uncached."""
    __slots__ = ("key", "value", "tensors", "made_on", "mark", "told", "kept")

    def __init__(self, key, value, tensors):
        self.key, self.value, self.tensors = key, value, list(tensors)
        self.made_on = self.mark = None
        self.told, self.kept = (), True
        first = self.tensors[0]
        if not first.is_cuda:
            return
        if torch.cuda.is_current_stream_capturing():
            self.kept = False
            return
        self.made_on = stream_of(first)
        at = (first.get_device(), self.made_on)
        self.mark = _marks.get(at) or _marks.setdefault(at, _Mark(first.device))
        self.mark.due = True

    def get(self):
        """The value, safe to use on the current stream; None where it cannot be made so (the stream it was made on is being captured)."""
        if self.made_on is not None:
            raw = stream_of(self.tensors[0])
            if raw != self.made_on and raw not in self.told and not torch.cuda.is_current_stream_capturing():
                with _capture_lock:                                   # no capture of this library's begins on that stream meanwhile
                    if self.mark.due:
                        with torch.cuda.stream(self.mark.stream):
                            if torch.cuda.is_current_stream_capturing():
                                return None
                        self.mark.record()
                here = torch.cuda.current_stream(self.tensors[0].device)
                here.wait_event(self.mark.event)
                for t in self.tensors:
                    t.record_stream(here)
                self.told += (raw,)
        return self.value

    def keep(self, old):
        """What to store: this, or the cache as it was."""
        return self if self.kept else old

    def __deepcopy__(self, memo):
        return None

    def __reduce__(self):
        return type(None), ()


@contextlib.contextmanager
def warm_up(stream: torch.cuda.Stream):
    """A pass ahead of a capture, on the stream that will capture: library workspaces, cached constants. One thread at a time (the
    lock graph_capture takes as well), so hold it over both."""
    with _capture_lock:
        here = torch.cuda.current_stream()
        stream.wait_stream(here)
        with torch.cuda.stream(stream):
            yield
        here.wait_stream(stream)


@contextlib.contextmanager
def graph_capture(graph, stream: torch.cuda.Stream | None = None, pool=None):
    """What the block launches goes into `graph`. One capture at a time in the process, in CUDA's thread-local mode: another
    thread may launch, allocate and synchronise its stream meanwhile (in torch's default mode its first cudaMalloc invalidates the
    capture), and no device-wide synchronisation or emptying of the allocator's cache on the way in, which stalls every other stream.

    The cyclic garbage collector stays off until the capture ends: a CUDAGraph of an earlier model that it frees in the middle
    destroys its executable graph, which CUDA refuses while the thread is capturing, and the capture is invalidated."""
    with _capture_lock:
        was_enabled = gc.isenabled()
        gc.disable()
        here, stream = torch.cuda.current_stream(), stream or torch.cuda.Stream()
        stream.wait_stream(here)
        try:
            with torch.cuda.stream(stream):
                graph.capture_begin(**({} if pool is None else dict(pool=pool)), capture_error_mode="thread_local")
                try:
                    yield
                except BaseException:
                    with contextlib.suppress(RuntimeError):           # the block's own error is the one to see
                        graph.capture_end()
                    raise
                graph.capture_end()
            here.wait_stream(stream)
        finally:
            if was_enabled:
                gc.enable()
