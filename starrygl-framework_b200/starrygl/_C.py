"""ctypes binding of libsgl_b200.so (the C ABI declared in include/sgl_b200.h).

There is no fallback: if the shared library is missing, or a tensor is not on a CUDA device, the call
raises.  ctypes releases the GIL around every foreign call, so the functions here can be driven from
worker threads the way the reference's pybind module is (csrc/srcs/starrygl/export.cu:193-250 uses
``py::gil_scoped_release`` on every heavy binding).
"""
import ctypes as C
import importlib.util
import os
import sys
import threading

import torch

_PKG_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB_PATH = os.path.join(_PKG_ROOT, "lib", "libsgl_b200.so")
HOST_PATH = os.path.join(_PKG_ROOT, "lib", f"_sgl_host.{torch.__version__}.{sys.implementation.cache_tag}.so")     # (as build.host_path)

SGL_DEV_BITS = {1: "node id out of range", 2: "timestamp outside the declared window", 4: "row index out of range",
                8: "output capacity exceeded", 16: "device-side wait timed out",
                32: "a peer sent a different number of rows than announced"}
POLICY = {"recent": 0, "uniform": 1}
GATHER_MODE = {"auto": 0, "vec": 1, "bulk": 2}

_lib = _host = None
_lock = threading.RLock()

_vp, _i64, _i32, _u64, _u32, _sz = C.c_void_p, C.c_int64, C.c_int, C.c_uint64, C.c_uint32, C.c_size_t

_SIGNATURES = {
    "sgl_last_error": (C.c_char_p, []),
    "sgl_build_info": (C.c_char_p, []),
    "sgl_radix_sort_ws_bytes": (_sz, [_i64]),
    "sgl_radix_sort_launches": (_i32, [_i64, _i32]),
    "sgl_radix_sort_u64_u32": (_i32, [_vp, _vp, _vp, _vp, _i64, _i32, C.POINTER(C.c_int), _vp, _sz, _vp]),
    "sgl_launch_graphs": (_i32, []),
    "sgl_look_back_limit": (_i64, [_i64]),
    "sgl_tcsr_build_ws_bytes": (_sz, [_i64, _i64]),
    "sgl_tcsr_build": (_i32, [_i64, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, C.POINTER(C.c_int64), _vp, _sz, _vp]),
    "sgl_tcsr_build_fenced": (_i32, [_i64, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, C.POINTER(C.c_int64), _vp, _sz,
                                     _vp]),
    "sgl_sample_ws_bytes": (_sz, [_i64]),
    "sgl_sample_layer": (_i32, [_vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _vp, _i32, _i32, _i32, _i64, _i32, _u64, _u32,
                                _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp]),
    "sgl_tcsr_fence_len": (_i64, [_i64, _i64]),
    "sgl_tcsr_fence": (_i32, [_vp, _vp, _i64, _i64, _vp, _vp]),
    "sgl_sample_layer_fenced": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _vp, _i32, _i32, _i32, _i64, _i32, _u64, _u32,
                                       _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp]),
    "sgl_sample_layer_counted": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _vp, _i32, _i32, _i32, _i64, _i32, _u64,
                                         _u32, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp, _i64, _vp]),
    "sgl_draws_below": (_i32, [_i64, _i32, _u32, _u64, _vp, _i64, _vp, _vp]),
    "sgl_sample_layer_static": (_i32, [_vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _i32, _i32, _i32, _i64, _i32, _u64, _u32,
                                       _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp]),
    "sgl_sample_gather": (_i32, [_vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _i32, _i32, _i32, _i64, _i32, _u64, _u32,
                                 _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _vp, _i32, _vp, _vp, _sz, _vp]),
    "sgl_sample_gather_fenced": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _i32, _i32, _i32, _i64, _i32, _u64, _u32,
                                        _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _vp, _i32, _vp, _vp, _sz, _vp]),
    "sgl_prefetch_batch": (_i32, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _i32, _i32, _i32, _i64, _i32, _u64, _u32,
                                  _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _vp, _i32, _vp, _vp, _sz, _vp, _i64, _vp, _vp]),
    "sgl_unique_pairs_ws_bytes": (_sz, [_i64]),
    "sgl_unique_pairs": (_i32, [_vp, _vp, _i64, _vp, _vp, _vp, _i64, _vp, _i32, _i32, _i64, _vp, _vp, _vp, _vp, _vp, _vp,
                                _vp, _sz, _vp]),
    "sgl_build_csc_ws_bytes": (_sz, [_i64, _i64]),
    "sgl_build_csc": (_i32, [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _vp, _i64, _vp, _i32, _i32, _i64, _vp, _vp, _vp, _vp, _vp,
                             _i32, _vp, _vp, _sz, _vp]),
    "sgl_relabel_nodes_ws_bytes": (_sz, [_i64]),
    "sgl_relabel_nodes": (_i32, [_vp, _i64, _vp, _i64, _vp, _vp, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp]),
    "sgl_gather_rows": (_i32, [_vp, _i64, _i64, _i64, _vp, _vp, _i64, _i64, _vp, _vp, _i64, _vp, _vp, _i32, _vp, _vp]),
    "sgl_cache_gather_ws_bytes": (_sz, [_i64]),
    "sgl_cache_gather": (_i32, [_vp, _i64, _vp, _i64, _vp, _i64, _vp, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp]),
    "sgl_scatter_rows": (_i32, [_vp, _i64, _i64, _i64, _vp, _vp, _i64, _i64, _vp, _vp, _i64, _vp, _vp, _i32, _vp, _vp]),
    "sgl_wire_pitch": (_i64, [_i64, _i32, _i32]),
    "sgl_route_pack": (_i32, [_vp, _i64, _i64, _vp, _vp, _vp, _i64, _vp, _vp, _vp]),
    "sgl_route_unpack": (_i32, [_vp, _i64, _i64, _vp, _i64, _i64, _vp, _vp, _vp]),
    "sgl_comm_unique_id": (_i32, [C.c_char_p, _sz]),
    "sgl_comm_init": (_i32, [C.POINTER(C.c_void_p), _i32, _i32, C.c_char_p]),
    "sgl_comm_destroy": (_i32, [_vp]),
    "sgl_route_exchange": (_i32, [_vp, _vp, C.POINTER(C.c_int64), _vp, C.POINTER(C.c_int64), _i64, _vp]),
    "sgl_cache_route_step": (_i32, [_vp, _vp, _i64, _i64, _vp, _vp, _vp, C.POINTER(C.c_int64), C.POINTER(C.c_int64), _vp,
                                    _vp, _vp, _i64, _vp, _i32, _vp, _vp]),
    "sgl_p2p_buffer_bytes": (_sz, [_i32, _i32, _i64, _i64]),
    "sgl_p2p_alloc": (_i32, [_sz, C.POINTER(C.c_void_p), C.c_char_p, _sz]),
    "sgl_p2p_open": (_i32, [C.c_char_p, C.POINTER(C.c_void_p)]),
    "sgl_p2p_close": (_i32, [_vp]),
    "sgl_p2p_free": (_i32, [_vp]),
    "sgl_p2p_route_create": (_i32, [_i32, _i32, _i32, _i64, _i64, C.POINTER(C.c_void_p), C.POINTER(C.c_void_p)]),
    "sgl_p2p_route_destroy": (_i32, [_vp]),
    "sgl_p2p_route_send": (_i32, [_vp, _vp, _i64, _i64, _vp, _vp, _vp, C.POINTER(C.c_int64), _u64, _vp, _vp]),
    "sgl_p2p_route_recv": (_i32, [_vp, C.POINTER(C.c_int64), _vp, _i64, _i64, _i32, _vp, _u64, _vp, _vp]),
    "sgl_densify_time_groups": (_i32, [_vp, _vp, _vp, _i64, _vp, _i64, _i64, _vp, _vp, _vp, _vp]),
    "sgl_comm_info": (_i32, [_vp, C.POINTER(C.c_int), C.POINTER(C.c_int)]),
    "sgl_init_p2p": (_i32, [C.POINTER(C.c_int), _i32, C.POINTER(C.c_int)]),
    "sgl_route_add_grouped": (_i32, [_vp, _i64, _i64, _vp, _vp, _vp, _i64, _vp, _i64, _vp, _vp]),
    "sgl_shard_gather": (_i32, [_vp, _vp, _i32, _i64, _vp, _i64, _vp, _vp, _vp, _vp]),
    "sgl_p2p_route_configure": (_i32, [_vp, _i64, _i64]),
    "sgl_p2p_route_send_dev": (_i32, [_vp, _vp, _i64, _i64, _vp, _vp, _vp, _vp, _i64, _u64, _vp, _vp]),
    "sgl_p2p_route_recv_dev": (_i32, [_vp, _i64, _vp, _i64, _i64, _i32, _vp, _u64, _vp, _vp]),
    "sgl_p2p_route_step": (_i32, [_vp, _vp, _i64, _i64, _vp, _vp, _vp, C.POINTER(C.c_int64), C.POINTER(C.c_int64), _vp, _i64,
                                  _vp, _u64, _vp, _vp]),
    "sgl_route_add_rows": (_i32, [_vp, _i64, _i64, _vp, _vp, _i64, _vp, _vp]),
    "sgl_dist_pack": (_i32, [_vp, _vp, _vp, _i64, _vp, _vp]),
    "sgl_dist_unpack": (_i32, [_vp, _i64, _vp, _vp, _vp, _vp]),
    "sgl_seeds_ws_bytes": (_sz, [_i64]),
    "sgl_seeds_in_window": (_i32, [_vp, _vp, _vp, _i64, _vp, _vp, _i64, _i64, _i32, _i32, _i64, _vp, _vp, _vp, _vp, _vp,
                                   _vp, _vp, _vp, _sz, _vp]),
    "sgl_lower_bound_i64": (_i32, [_vp, _i64, _vp, _i32, _vp, _vp]),
    "sgl_plan_route_ws_bytes": (_sz, [_i64, _i64]),
    "sgl_plan_route": (_i32, [_vp, _i64, _vp, _vp, _i64, _i64, _vp, _vp, _vp, _i64, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _vp,
                              _sz, _vp]),
    "sgl_plan_routes_ws_bytes": (_sz, [_i32, _vp, _vp]),
    "sgl_plan_routes": (_i32, [_i32, _vp, _vp, _vp, _vp, _i64, _i64, _vp, _vp, _vp, _i64, _vp, _vp, _vp, _vp, _vp, _sz, _vp]),
    "sgl_slice_window_ws_bytes": (_sz, [_i64]),
    "sgl_slice_window": (_i32, [_vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _i64, _i64, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _vp,
                                _vp, _vp, _vp, _sz, _vp]),
    "sgl_copy_prefix": (_i32, [_i32, _vp, _vp, _vp, _vp, _i64, _vp]),
    "sgl_mail_reduce_ws_bytes": (_sz, [_i64]),
    "sgl_mail_reduce": (_i32, [_vp, _i64, _vp, _i64, _i64, _vp, _i64, _i32, _i32, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp,
                               _sz, _vp]),
    "sgl_mail_reduce_counted": (_i32, [_vp, _i64, _vp, _i64, _i64, _vp, _i64, _i32, _i32, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp,
                                       _vp, _sz, _vp, _i64, _vp]),
    "sgl_mailbox_write": (_i32, [_vp, _i64, _vp, _vp, _vp, _i64, _vp, _vp, _vp, _i64, _i64, _i32, _vp, _vp]),
    "sgl_build_batch_layout": (_i64, [_i64, _vp, _i32, _vp]),
    "sgl_build_batch_ws_bytes": (_sz, [_i64, _vp, _i32]),
    "sgl_build_batch": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _vp, _i32, _i32, _i32, _i64, _u64, _i32, _i32, _i64,
                               _vp, _vp, _vp, _vp, _vp, _sz, _vp, _vp]),
    "sgl_build_batch_at": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _vp, _i32, _i32, _i32, _i64, _u64, _i32, _i32, _i64,
                                  _vp, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp, _vp]),
    "sgl_build_batch_staged": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _vp, _i32, _i32, _i32, _i64, _u64, _i32, _i32, _i64,
                                      _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp, _vp]),
    "sgl_build_batch_ready": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _i64, _vp, _i32, _i32, _i32, _i64, _u64, _i32, _i32, _i64,
                                     _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp, _vp]),
    "sgl_query_layout": (_i64, [_i64, _i64, _i32, _i32, _vp]),
    "sgl_query_ws_bytes": (_sz, [_i64, _i64, _i32, _i32]),
    "sgl_query": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _vp, _vp, _i64, _vp, _vp, _i64, _i32, _i32,
                         _i32, _i32, _i64, _i32, _i32, _i32, _i64, _vp, _vp, _i64, _i32, _vp, _vp, _vp, _vp, _vp, _sz, _vp, _vp]),
    "sgl_query_at": (_i32, [_vp, _vp, _vp, _vp, _vp, _i64, _vp, _vp, _vp, _i64, _i64, _i64, _i64, _vp, _vp, _i64, _vp, _vp, _i64, _i32, _i32,
                         _i32, _i32, _i64, _i32, _i32, _i32, _i64, _vp, _vp, _i64, _i32, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp, _vp]),
    "sgl_query_blocks": (_i32, [_i32, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _vp, _vp]),
    "sgl_export_arrays": (_i32, [_i32, _vp, _vp, _vp, _vp, _vp, _i64, _vp, _i64, _vp]),
    "sgl_copy_arrays": (_i32, [_i32, _vp, _vp, _vp, _vp]),
    "sgl_host_words": (_i32, [C.POINTER(C.c_void_p)]),
    "sgl_wait_word": (_i32, [_vp, _i64, _vp]),
    "sgl_read_back": (_i32, [_vp, _vp, _sz, _vp]),
    "sgl_graph_capture_begin": (_i32, [_vp]),
    "sgl_graph_capture_end": (_i32, [_vp, C.POINTER(C.c_void_p)]),
    "sgl_graph_launch": (_i32, [_vp, _vp, _vp, _sz, _vp]),
    "sgl_graph_destroy": (_i32, [_vp]),
    "sgl_replica_lookup_ws_bytes": (_sz, [_i64]),
    "sgl_replica_lookup": (_i32, [_vp, _vp, _vp, _i64, _vp, _i64, _i64, _vp, _vp, _vp, _vp, _vp, _vp, _sz, _vp]),
}


def lib():
    """The loaded shared library; raises if it has not been built."""
    global _lib
    if _lib is None:
        with _lock:
            if _lib is None:
                if not os.path.exists(LIB_PATH):
                    raise RuntimeError(
                        f"{LIB_PATH} is missing: build it with `python starrygl-framework_b200/build.py` "
                        "(there is no CPU or PyTorch fallback for these operators)")
                l = C.CDLL(LIB_PATH)
                for name, (res, args) in _SIGNATURES.items():
                    f = getattr(l, name)
                    f.restype, f.argtypes = res, args
                _lib = l
    return _lib


class SglError(RuntimeError):
    pass


def host():
    """The extension module over the same library (csrc/host.cpp) for the calls that every mini-batch makes: its functions take tensors
    and integers, raise by themselves, and cost a fraction of a ctypes call."""
    global _host
    if _host is None:
        with _lock:
            if _host is None:
                lib()
                if not os.path.exists(HOST_PATH):
                    raise RuntimeError(f"{HOST_PATH} is missing: build it for this torch with `python starrygl-framework_b200/build.py`")
                spec = importlib.util.spec_from_file_location("_sgl_host", HOST_PATH)
                m = importlib.util.module_from_spec(spec)
                spec.loader.exec_module(m)
                m.bind(SglError, sys.modules[__name__])
                _host = m
    return _host


def check(rc):
    if rc != 0:
        raise SglError(f"libsgl_b200 error {rc}: {lib().sgl_last_error().decode()}")


def ptr(t):
    """Device-usable pointer of a tensor (None -> NULL): CUDA memory, or pinned host memory, which the GPU
    addresses directly under unified addressing.  Pageable CPU tensors are refused: there is no CPU path."""
    if t is None:
        return None
    if not t.is_cuda and not t.is_pinned():
        raise SglError("expected a CUDA (or pinned host) tensor: the data path has no CPU implementation")
    if not t.is_contiguous():
        raise SglError("expected a contiguous tensor")
    return t.data_ptr()


def stream_ptr(stream=None):
    if stream is not None:
        return stream.cuda_stream
    if torch.cuda.is_initialized():     # a tenth of the cost of building a Stream object
        return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())
    return torch.cuda.current_stream().cuda_stream


_STREAMS = {}


def current_stream(device=None):
    """torch.cuda.current_stream(device) with the Stream objects kept (by stream, as many as a program has)."""
    index = None if device is None else device.index
    key = torch._C._cuda_getCurrentStream(torch._C._cuda_getDevice() if index is None else index)
    s = _STREAMS.get(key)
    if s is None:
        if len(_STREAMS) >= 256:
            _STREAMS.clear()
        s = _STREAMS[key] = torch.cuda.Stream(stream_id=key[0], device_index=key[1], device_type=key[2])
    return s


class on_stream:
    """``with torch.cuda.stream(s)`` for a stream of the current device, at a fifth of its cost (other devices: that)."""

    def __init__(self, stream):
        self._to, self._slow = stream, None

    def __enter__(self):
        s = self._to
        if torch._C._cuda_getDevice() != s.device_index:
            self._slow = torch.cuda.stream(s)
            return self._slow.__enter__()
        self._from = torch._C._cuda_getCurrentStream(s.device_index)
        torch._C._cuda_setStream(stream_id=s.stream_id, device_index=s.device_index, device_type=s.device_type)

    def __exit__(self, *exc):
        if self._slow is not None:
            return self._slow.__exit__(*exc)
        i, d, t = self._from
        torch._C._cuda_setStream(stream_id=i, device_index=d, device_type=t)


_HOST = threading.local()


def host_words():
    """(address, ctypes int64 array) of the calling thread's pinned result buffer."""
    h = _HOST.__dict__.get("words")
    if h is None:
        p = C.c_void_p()
        check(lib().sgl_host_words(C.byref(p)))
        h = _HOST.__dict__["words"] = (p.value, (C.c_int64 * 512).from_address(p.value))
    return h


def abandon():
    """A call that fails behind its launches waits for the current stream: what is still running writes to the thread's result words, and the
    thread's next call would take it for its own.  (A capturing stream runs nothing.)"""
    try:
        if not torch._C._cuda_isCurrentStreamCapturing():
            current_stream().synchronize()
    except RuntimeError:
        pass                             # (the call's own error says more)


class CountRing:
    """Pinned (value, sequence number) pairs that kernels fill in with a count the host may ask for later.  A pair is used
    again after as many calls as there are pairs, once its count has arrived -- so that one kernel at a time may write to it;
    who still wants the older count reads it from the device."""
    SLOTS = 1024

    def __init__(self):
        self._seq = 0
        self._lock = threading.Lock()
        self._buf = self._words = None
        self._owner = [0] * self.SLOTS       # sequence number the pair was last given out for

    def take(self):
        """(address, index of the value, sequence number); None while the pair's last count is still on its way."""
        with self._lock:
            if self._buf is None:
                buf = torch.zeros(2 * self.SLOTS, dtype=torch.int64).pin_memory()
                self._words = (C.c_int64 * (2 * self.SLOTS)).from_address(buf.data_ptr())
                self._base, self._buf = buf.data_ptr(), buf
            seq = self._seq = self._seq + 1
            k = seq % self.SLOTS
            if self._words[2 * k + 1] != self._owner[k]:
                return None
            self._owner[k] = seq
        return self._base + 16 * k, 2 * k, seq

    def give_back(self, taken):
        """The pair of a call that failed: nothing is going to arrive."""
        if taken is not None:
            self._words[taken[1] + 1] = taken[2]

    def value(self, taken, stream):
        """The count, or None when its pair was used again (or never filled in)."""
        addr, i, seq = taken
        w = self._words
        if self._owner[i // 2] != seq:
            return None
        if w[i + 1] < seq:
            lib().sgl_wait_word(addr + 8, seq, stream)
        arrived, v = w[i + 1] == seq, w[i]
        return v if arrived and self._owner[i // 2] == seq else None     # (given out again meanwhile: v may be the next one's)


COUNTS = CountRing()


def read_words(t, count):
    """The first ``count`` int64 words of a device tensor, as a list (waits for the current stream's work on them)."""
    buf = (C.c_int64 * count)()
    host().sgl_read_back(t.data_ptr(), C.addressof(buf), 8 * count, stream_ptr())
    return list(buf)


class Workspace:
    """Per-(device, stream) scratch buffer handed to the library; grows geometrically, never shrinks."""

    def __init__(self):
        self._bufs = {}

    def get(self, nbytes, device, stream_id):
        key = (device.index, stream_id)
        b = self._bufs.get(key)
        if b is None or b.numel() < nbytes:
            b = torch.empty(max(int(nbytes * 1.25), 1 << 16), dtype=torch.uint8, device=device)
            self._bufs[key] = b
        return b


WORKSPACE = Workspace()


def workspace(nbytes, device, stream=None):
    sp = stream_ptr(stream)
    b = WORKSPACE.get(nbytes, device, sp)
    return b, b.data_ptr(), b.numel()


def decode_status(v):
    return ", ".join(txt for bit, txt in SGL_DEV_BITS.items() if v & bit) or "ok"
