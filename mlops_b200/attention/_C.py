"""Binding of the C library (include/mlops_fbla.h) for PyTorch tensors: the four functions of the reference's compiled
`mlops.attention._C` module (attention/python/csrc/mlops_attention_torch.cpp:99-111), same names, argument orders,
checks and exceptions -- scratch_bytes, images_bytes, decode, prefill. PyTorch supplies device memory and the current
stream only; every computation happens inside libmlops_attention.so. There is no CPU fallback: importing this module
without the built library raises."""
import collections
import ctypes
import functools
import os
import threading

import torch

_LIB_PATH = os.environ.get("MLOPS_FBLA_LIBRARY") or os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lib",
                                                                  "libmlops_attention.so")
if not os.path.exists(_LIB_PATH):
    raise ImportError(f"{_LIB_PATH} is missing: build it with `make -C mlops_b200/csrc` (or __graft_entry__.build()); "
                      "this package has no fallback path")
_lib = ctypes.CDLL(_LIB_PATH)

__version__ = "0.4.0"
OK, INVALID_VALUE, CUDA_ERROR = 0, 1, 2


class Config(ctypes.Structure):
    """mlops_fbla_config (64 bytes)."""
    _fields_ = [("batch", ctypes.c_int), ("q_heads", ctypes.c_int), ("kv_heads", ctypes.c_int), ("tokens", ctypes.c_int),
                ("scale", ctypes.c_float), ("tau", ctypes.c_float), ("format", ctypes.c_int), ("capacity", ctypes.c_int),
                ("head_stride", ctypes.c_int), ("group_stride", ctypes.c_int),
                ("out_head_stride", ctypes.c_int64), ("out_token_stride", ctypes.c_int64),
                ("length_stride", ctypes.c_int)]


class Cache(ctypes.Structure):
    """mlops_fbla_cache (64 bytes)."""
    _fields_ = [(n, ctypes.c_void_p) for n in ("coarse", "fine", "meta", "exact_sink_k", "exact_sink_v", "exact_open_k",
                                               "exact_open_v", "tc_images")]


class Sizes(ctypes.Structure):
    _fields_ = [(n, ctypes.c_size_t) for n in ("coarse", "fine", "meta", "exact", "images")]


_vp, _cp = ctypes.c_void_p, ctypes.POINTER(Config)
_lib.mlops_fbla_decode_scratch_bytes.restype = ctypes.c_size_t
_lib.mlops_fbla_decode_scratch_bytes.argtypes = [_cp]
_lib.mlops_fbla_decode_scratch_bytes_for.restype = ctypes.c_size_t
_lib.mlops_fbla_decode_scratch_bytes_for.argtypes = [_cp, ctypes.c_int]
_lib.mlops_fbla_images_bytes.restype = ctypes.c_size_t
_lib.mlops_fbla_images_bytes.argtypes = [_cp]
_lib.mlops_fbla_cache_sizes.restype = ctypes.c_int
_lib.mlops_fbla_cache_sizes.argtypes = [_cp, ctypes.POINTER(Sizes)]
_lib.mlops_fbla_decode.restype = ctypes.c_int
_lib.mlops_fbla_decode.argtypes = [_cp, _vp, ctypes.POINTER(Cache), _vp, _vp, ctypes.c_size_t, _vp]
_lib.mlops_fbla_decode_at.restype = ctypes.c_int
_lib.mlops_fbla_decode_at.argtypes = [_cp, _vp, _vp, ctypes.POINTER(Cache), _vp, _vp, ctypes.c_size_t, _vp]
_lib.mlops_fbla_prefill.restype = ctypes.c_int
_lib.mlops_fbla_prefill.argtypes = [_cp, ctypes.c_int, _vp, _vp, _vp, ctypes.POINTER(Cache), _vp, _vp]
_lib.mlops_fbla_encode.restype = ctypes.c_int
_lib.mlops_fbla_encode.argtypes = [_cp, ctypes.c_int, _vp, _vp, ctypes.POINTER(Cache), _vp]
_lib.mlops_fbla_prefill_at.restype = ctypes.c_int
_lib.mlops_fbla_prefill_at.argtypes = [_cp, _vp, _vp, ctypes.c_int, _vp, _vp, _vp, ctypes.POINTER(Cache), _vp, _vp]
_lib.mlops_fbla_append_at.restype = ctypes.c_int
_lib.mlops_fbla_append_at.argtypes = [_cp, _vp, _vp, _vp, ctypes.POINTER(Cache), _vp]
_lib.mlops_fbla_last_error.restype = ctypes.c_char_p
_lib.mlops_fbla_status_string.restype = ctypes.c_char_p
_lib.mlops_fbla_status_string.argtypes = [ctypes.c_int]

lib = _lib  # the raw C ABI, for callers that drive it directly (tests, the bench)


def last_error():
    return _lib.mlops_fbla_last_error().decode()


def _raise(status, what):
    if status == INVALID_VALUE:
        raise ValueError(last_error())
    if status != OK:
        raise RuntimeError(f"{what} failed: {last_error()}")


def _config(batch, q_heads, kv_heads, tokens, fmt, capacity, scale, tau):
    if fmt not in (0, 1):
        raise ValueError("format must be 0 (3+3) or 1 (4+2)")
    return Config(int(batch), int(q_heads), int(kv_heads), int(tokens), float(scale), float(tau), int(fmt), int(capacity), 0, 0, 0, 0, 0)


def _tensor(x, dev, dtype, what):
    if not x.is_cuda or x.device != dev:
        raise ValueError(f"{what}: expected a CUDA tensor on {dev}")
    if x.dtype != dtype or not x.is_contiguous():
        raise ValueError(f"{what}: expected a contiguous {dtype} tensor")


def _cache(coarse, fine, meta, sk, sv, ok, ov, images=None):
    return Cache(coarse.data_ptr(), fine.data_ptr(), meta.data_ptr(), sk.data_ptr(), sv.data_ptr(), ok.data_ptr(), ov.data_ptr(),
                 images.data_ptr() if images is not None else None)


def _stream(dev):
    return ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)


def scratch_bytes(batch, q_heads, kv_heads, tokens, format, capacity):
    """Bytes of scratch one decode needs on the current device."""
    cfg = _config(batch, q_heads, kv_heads, tokens, format, capacity, 0.0, 0.0)
    n = int(_lib.mlops_fbla_decode_scratch_bytes(ctypes.byref(cfg)))
    if n <= 0:
        raise ValueError(f"invalid FBLA configuration: batch {batch}, heads {q_heads} / {kv_heads}, tokens {tokens}, capacity {capacity}")
    return n


# ---- calls on a whole cache object --------------------------------------------------------------------------------------------
_U8, _BF16 = torch.uint8, torch.bfloat16


def _arrays(c):
    """A cache's arrays, checked as `decode` and `prefill` check theirs: the structure that names them to the library, their device's index.
    (Looked at in every call -- 3 us of the host's time -- and nothing of it kept: a cache is a plain record that its user may change,
    copy and save.)"""
    k, f, m, sk, sv, ok, ov = c.coarse, c.fine, c.meta, c.sink_k, c.sink_v, c.open_k, c.open_v
    index = k.get_device()
    if not (0 <= index == f.get_device() == m.get_device() == sk.get_device() == sv.get_device() == ok.get_device() == ov.get_device()
            and k.dtype is f.dtype is _U8 and m.dtype is sk.dtype is sv.dtype is ok.dtype is ov.dtype is _BF16
            and k.is_contiguous() and f.is_contiguous() and m.is_contiguous() and sk.is_contiguous() and sv.is_contiguous()
            and ok.is_contiguous() and ov.is_contiguous()):
        for x in (k, f):
            _tensor(x, k.device, _U8, "packed cache records")
        for x in (m, sk, sv, ok, ov):
            _tensor(x, k.device, _BF16, "cache metadata / exact group")
    images = c.images
    return Cache(k.data_ptr(), f.data_ptr(), m.data_ptr(), sk.data_ptr(), sv.data_ptr(), ok.data_ptr(), ov.data_ptr(),
                 images.data_ptr() if images is not None else None), index


def _rows(x, index, what):
    """as _tensor, for a BF16 operand on the cache's device"""
    if x.get_device() != index or x.dtype is not _BF16 or not x.is_contiguous():
        _tensor(x, torch.device("cuda", index), _BF16, what)


_scratch_bytes = functools.lru_cache(maxsize=256)(lambda device, *shape: scratch_bytes(*shape))
_raw_stream = torch._C._cuda_getCurrentRawStream
_capturing = torch._C._cuda_isCurrentStreamCapturing


class _Scratch:
    """a decode's scratch; `lock` is held while a call's kernels are enqueued, so that threads on one stream do not mix theirs"""
    __slots__ = ("bytes", "buffer", "pointer", "lock")

    def __init__(self, nbytes, device):
        self.bytes, self.lock = nbytes, threading.Lock()
        self.buffer = torch.empty((nbytes,), dtype=torch.uint8, device=device)  # the library needs no initial contents
        self.pointer = self.buffer.data_ptr()


class _ScratchPool:
    """Decode scratch, one buffer per (device, stream), grown on demand and kept for later calls -- at most BUFFERS of them, the
    least recently used one given back first (to the stream's own free memory: the kernels that use it come before whatever takes it
    next). Calls of one stream run in order, so they may share one; calls of different streams never do. A call that is being captured
    has one of its own, from the graph's memory: a replay may run on any stream and at any later time."""
    BUFFERS = 16

    def __init__(self):
        self._held, self._lock = collections.OrderedDict(), threading.Lock()

    def get(self, device, stream, nbytes):
        if device.type == "cuda" and _capturing():
            return _Scratch(nbytes, device)
        key = device, stream
        with self._lock:
            held = self._held.get(key)
            if held is not None and held.bytes >= nbytes:
                self._held.move_to_end(key)
                return held
            self._held[key] = held = _Scratch(nbytes, device)
            self._held.move_to_end(key)
            while len(self._held) > self.BUFFERS:
                self._held.popitem(last=False)
        return held


_pool = _ScratchPool()


def decode_cache(q, c, scale, tau):
    """decode of a whole cache object with the pool's scratch"""
    struct, index = _arrays(c)
    if q.dim() != 3 or q.size(2) != 128:
        raise ValueError(f"q must be [batch, q_heads, 128], got {tuple(q.shape)}")
    if not q.is_contiguous():
        q = q.contiguous()
    if q.get_device() != index:
        raise ValueError(f"q: expected a CUDA tensor on cuda:{index}")
    if torch._C._cuda_getDevice() != index:
        with torch.cuda.device(index):
            return decode_cache(q, c, scale, tau)
    batch, q_heads, kv_heads = q.size(0), q.size(1), c.meta.size(1)
    tokens, capacity = int(c.tokens), int(c.capacity)
    room = min(capacity, -(-tokens // 16384) * 16384)  # (asked for once in 16 384 tokens; a slot may have room for far more than it holds)
    need = _scratch_bytes(index, batch, q_heads, kv_heads, room, c.format, capacity)
    stream = _raw_stream(index)
    scratch = _pool.get(q.device, stream, need)
    out = torch.empty_like(q)
    cfg = Config(batch, q_heads, kv_heads, tokens, float(scale), float(tau), int(c.format), capacity, 0, 0, 0, 0, 0)
    with scratch.lock:
        status = _lib.mlops_fbla_decode(ctypes.byref(cfg), q.data_ptr(), ctypes.byref(struct), out.data_ptr(), scratch.pointer, scratch.bytes, stream)
    _raise(status, "mlops_fbla_decode")
    return out


def prefill_cache(q, k, v, c, scale):
    """prefill (append for q None) on a whole cache object; k and v contiguous BF16 of the cache's batch and KV heads"""
    struct, index = _arrays(c)
    _rows(k, index, "k")
    _rows(v, index, "v")
    if torch._C._cuda_getDevice() != index:
        with torch.cuda.device(index):
            return prefill_cache(q, k, v, c, scale)
    batch, kv_heads, n, out = c.meta.size(0), c.meta.size(1), k.size(2), None
    q_heads = kv_heads
    if q is not None:
        if q.dim() != 4 or q.size(0) != batch or q.size(2) != n or q.size(3) != 128:
            raise ValueError(f"q must be [batch, q_heads, n, 128] matching k, got {tuple(q.shape)}")
        _rows(q, index, "q")
        q_heads, out = q.size(1), torch.empty_like(q)
    cfg = Config(batch, q_heads, kv_heads, int(c.tokens), float(scale), 0.0, int(c.format), int(c.capacity), 0, 0, 0, 0, 0)
    _raise(_lib.mlops_fbla_prefill(ctypes.byref(cfg), n, q.data_ptr() if q is not None else None, k.data_ptr(), v.data_ptr(), ctypes.byref(struct),
                                   out.data_ptr() if out is not None else None, _raw_stream(index)), "mlops_fbla_prefill")
    return out


def images_bytes(batch, kv_heads, capacity):
    """Bytes of persistent prefill images on the current device (this library keeps none: 0)."""
    cfg = _config(batch, kv_heads, kv_heads, 0, 0, capacity, 0.0, 0.0)
    return int(_lib.mlops_fbla_images_bytes(ctypes.byref(cfg)))


def decode(q, coarse, fine, meta, sink_k, sink_v, open_k, open_v, scratch, tokens, capacity, kv_heads, format, scale=0.0, tau=0.0):
    if q.dim() != 3 or q.size(2) != 128:
        raise ValueError(f"q must be [batch, q_heads, 128], got {tuple(q.shape)}")
    dev = q.device
    _tensor(q, dev, torch.bfloat16, "q")
    for x in (coarse, fine):
        _tensor(x, dev, torch.uint8, "packed cache records")
    for x in (meta, sink_k, sink_v, open_k, open_v):
        _tensor(x, dev, torch.bfloat16, "cache metadata / exact group")
    _tensor(scratch, dev, torch.uint8, "scratch")
    cfg = _config(q.size(0), q.size(1), kv_heads, tokens, format, capacity, scale, tau)
    cache = _cache(coarse, fine, meta, sink_k, sink_v, open_k, open_v)
    out = torch.empty_like(q)
    with torch.cuda.device(dev):
        st = _lib.mlops_fbla_decode(ctypes.byref(cfg), q.data_ptr(), ctypes.byref(cache), out.data_ptr(), scratch.data_ptr(),
                                    scratch.numel(), _stream(dev))
    _raise(st, "mlops_fbla_decode")
    return out


def prefill(q, k, v, coarse, fine, meta, sink_k, sink_v, open_k, open_v, tokens, capacity, q_heads, format, scale=0.0, images=None):
    """Appends k / v [B, Hkv, n, 128] to the cache holding `tokens`; with q [B, Hq, n, 128] returns the attention of
    every new position (None for q None: append only)."""
    if k.dim() != 4 or k.size(3) != 128 or v.shape != k.shape:
        raise ValueError(f"k and v must be [batch, kv_heads, n, 128], got {tuple(k.shape)} and {tuple(v.shape)}")
    dev = k.device
    _tensor(k, dev, torch.bfloat16, "k")
    _tensor(v, dev, torch.bfloat16, "v")
    for x in (coarse, fine):
        _tensor(x, dev, torch.uint8, "packed cache records")
    for x in (meta, sink_k, sink_v, open_k, open_v):
        _tensor(x, dev, torch.bfloat16, "cache metadata / exact group")
    B, Hkv, n = k.size(0), k.size(1), k.size(2)
    if q is not None:
        if q.dim() != 4 or q.size(0) != B or q.size(1) != q_heads or q.size(2) != n or q.size(3) != 128:
            raise ValueError(f"q must be [batch, q_heads, n, 128] matching k, got {tuple(q.shape)}")
        _tensor(q, dev, torch.bfloat16, "q")
    cfg = _config(B, q_heads, Hkv, tokens, format, capacity, scale, 0.0)
    cache = _cache(coarse, fine, meta, sink_k, sink_v, open_k, open_v, images)
    out = torch.empty_like(q) if q is not None else None
    with torch.cuda.device(dev):
        st = _lib.mlops_fbla_prefill(ctypes.byref(cfg), int(n), q.data_ptr() if q is not None else None, k.data_ptr(), v.data_ptr(),
                                     ctypes.byref(cache), out.data_ptr() if out is not None else None, _stream(dev))
    _raise(st, "mlops_fbla_prefill")
    return out


def encode(k, v, coarse, fine, meta, sink_k, sink_v, open_k, open_v, capacity, format):
    """Stores k / v [B, Hkv, n, 128], n > 0, into an empty cache for `capacity` tokens; its arrays need no initial contents."""
    dev = k.device
    _tensor(k, dev, torch.bfloat16, "k")
    _tensor(v, dev, torch.bfloat16, "v")
    if torch._C._cuda_getDevice() != dev.index:
        with torch.cuda.device(dev):
            return encode(k, v, coarse, fine, meta, sink_k, sink_v, open_k, open_v, capacity, format)
    cfg = _config(k.size(0), k.size(1), k.size(1), 0, format, capacity, 0.0, 0.0)
    cache = _cache(coarse, fine, meta, sink_k, sink_v, open_k, open_v)
    _raise(_lib.mlops_fbla_encode(ctypes.byref(cfg), k.size(2), k.data_ptr(), v.data_ptr(), ctypes.byref(cache), _raw_stream(dev.index)), "mlops_fbla_encode")
