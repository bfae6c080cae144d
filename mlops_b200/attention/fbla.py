"""The `mlops.attention` Python interface over the CUDA library.

The public surface is the reference's (attention/python/mlops/attention/fbla.py:43-150): the ``FBLACache`` record and
``empty / encode / append / prefill / decode`` with the same argument names, defaults and exception types, so code
written against `mlops.attention` runs unchanged. Shapes: K / V chunks ``[B, Hkv, n, 128]``, prefill queries
``[B, Hq, n, 128]``, decode queries ``[B, Hq, 128]``, all BF16 on one CUDA device. Everything that touches cache bytes
or computes attention happens inside libmlops_attention.so; this module only allocates tensors and forwards.
"""
from dataclasses import dataclass
from typing import Optional

import torch

from . import _C

GROUP = 128      # tokens per quantisation group
HEAD_DIM = 128
# mode string -> (coarse bits, fine bits, value of mlops_fbla_format)
_PLANES = {"3+3": (3, 3, 0), "4+2": (4, 2, 1)}


@dataclass
class FBLACache:
    coarse: torch.Tensor  # uint8  [B, Hkv, 8 * groups, 512 * coarse bits]: the coarse plane's records
    fine: torch.Tensor    # uint8  [B, Hkv, 8 * groups, 512 * fine bits]
    meta: torch.Tensor    # bf16   [B, Hkv, groups, 512]: per-channel base / step of K and V
    sink_k: torch.Tensor  # bf16   [B, Hkv, 128, 128]: the first group, kept exact
    sink_v: torch.Tensor
    open_k: torch.Tensor  # bf16   [B, Hkv, 128, 128]: the group still being filled
    open_v: torch.Tensor
    tokens: int
    capacity: int
    format: int
    images: Optional[torch.Tensor] = None  # the reference's persistent prefill images; this library has none


def _require_kv(k, v):
    """K and V of one chunk: equal 4-D shapes with a head dimension of 128, on one CUDA device."""
    shape = k.shape
    if not (len(shape) == 4 and shape == v.shape and shape[3] == HEAD_DIM):
        raise ValueError(f"expected k and v of one shape [B, Hkv, n, {HEAD_DIM}]; k is {tuple(k.shape)}, v is {tuple(v.shape)}")
    if not (k.is_cuda and v.is_cuda and k.get_device() == v.get_device()):
        raise ValueError(f"k and v have to live on the same CUDA device (k: {k.device}, v: {v.device})")


def _dense(x):
    """as the library reads K and V: BF16, contiguous"""
    return x if x.dtype is torch.bfloat16 and x.is_contiguous() else x.to(torch.bfloat16).contiguous()


def _allocate(make, like, batch, kv_heads, capacity, mode, device) -> FBLACache:
    """The arrays of a cache for ``capacity`` tokens, each from ``make(shape, dtype=, device=)`` or ``like(another)``."""
    planes = _PLANES.get(mode)
    if planes is None:
        raise ValueError(f"unknown mode {mode!r}: choose '3+3' or '4+2'")
    coarse_bits, fine_bits, fmt = planes
    groups = -(-capacity // GROUP)
    records = 8 * groups
    sink_k = make((batch, kv_heads, GROUP, HEAD_DIM), dtype=torch.bfloat16, device=device)
    sink_v, open_k, open_v = like(sink_k), like(sink_k), like(sink_k)
    return FBLACache(coarse=make((batch, kv_heads, records, 512 * coarse_bits), dtype=torch.uint8, device=device),
                     fine=make((batch, kv_heads, records, 512 * fine_bits), dtype=torch.uint8, device=device),
                     meta=make((batch, kv_heads, groups, 512), dtype=torch.bfloat16, device=device),
                     sink_k=sink_k, sink_v=sink_v, open_k=open_k, open_v=open_v, tokens=0, capacity=capacity, format=fmt)


def empty(batch: int, kv_heads: int, capacity: int, mode: str = "3+3", device="cuda") -> FBLACache:
    """A cache with room for ``capacity`` tokens and none stored. All arrays start as zeros."""
    cache = _allocate(torch.zeros, torch.zeros_like, batch, kv_heads, capacity, mode, device)
    with torch.cuda.device(torch.device(device)):
        image_bytes = _C.images_bytes(batch, kv_heads, -(-capacity // GROUP) * GROUP)
    if image_bytes > 0:
        cache.images = torch.zeros((image_bytes,), dtype=torch.uint8, device=device)
    return cache


def _extend(cache, k, v, q=None, scale=0.0):
    """One library call: store the chunk (k, v) behind the cache's tokens and, given q, attend from its positions."""
    _require_kv(k, v)
    meta, added = cache.meta, k.size(2)
    if k.size(0) != meta.size(0) or k.size(1) != meta.size(1):
        raise ValueError(f"the chunk is [batch, kv_heads] = {tuple(k.shape[:2])} but the cache was built for {tuple(meta.shape[:2])}")
    if cache.tokens + added > cache.capacity:
        raise ValueError(f"{added} more tokens do not fit: the cache holds {cache.tokens} of {cache.capacity}")
    result = _C.prefill_cache(q, _dense(k), _dense(v), cache, scale)
    cache.tokens += added
    return result


@torch.no_grad()
def encode(k: torch.Tensor, v: torch.Tensor, mode: str = "3+3", capacity: Optional[int] = None) -> FBLACache:
    """Quantise dense K / V ``[B, Hkv, N, 128]`` into a new cache (room for ``capacity`` tokens, default N)."""
    _require_kv(k, v)
    batch, kv_heads, n = (int(x) for x in k.shape[:3])
    room = n if capacity is None else int(capacity)
    if room < n:
        raise ValueError(f"a capacity of {room} tokens cannot hold the {n} given")
    if n == 0 or batch == 0 or kv_heads == 0:
        cache = empty(batch, kv_heads, room, mode, k.device)
        _extend(cache, k, v)
        return cache
    # (the call that stores the tokens also zeroes what they leave of the arrays)
    cache = _allocate(torch.empty, torch.empty_like, batch, kv_heads, room, mode, k.device)
    _C.encode(_dense(k), _dense(v), cache.coarse, cache.fine, cache.meta, cache.sink_k,
              cache.sink_v, cache.open_k, cache.open_v, room, cache.format)
    cache.tokens = n
    return cache


@torch.no_grad()
def append(cache: FBLACache, k: torch.Tensor, v: torch.Tensor) -> FBLACache:
    """Store ``[B, Hkv, n, 128]`` more K / V in ``cache`` (in place; also returned). Tokens land in the BF16 open
    group; once a group is full it is quantised when the following token arrives, so growing a cache token by token
    ends in the same bytes as :func:`encode` of the whole sequence."""
    _extend(cache, k, v)
    return cache


@torch.no_grad()
def prefill(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cache: FBLACache, *, scale: float = 0.0) -> torch.Tensor:
    """Causal attention of a chunk. ``k, v [B, Hkv, n, 128]`` are stored in ``cache`` first; the query of chunk
    position i (absolute position ``tokens + i``) sees every token up to its own. Returns ``[B, Hq, n, 128]`` BF16."""
    fits = q.dtype == torch.bfloat16 and q.ndim == 4 and k.ndim > 2 and q.size(0) == k.size(0) and q.size(2) == k.size(2)
    if not fits:
        raise ValueError(f"q has to be a bfloat16 [B, Hq, n, {HEAD_DIM}] tensor with the batch and length of k {tuple(k.shape)}; "
                         f"it is {q.dtype} {tuple(q.shape)}")
    return _extend(cache, k, v, q.contiguous(), scale)


def decode(q: torch.Tensor, cache: FBLACache, *, scale: float = 0.0, tau: float = 0.0) -> torch.Tensor:
    """Attention of one new query per head, ``q [B, Hq, 128]`` BF16, over everything in ``cache``.
    ``scale`` 0 selects 1/sqrt(128); ``tau`` 0 selects the format's refinement threshold."""
    if q.dtype != torch.bfloat16:
        raise TypeError(f"decode takes bfloat16 queries, not {q.dtype}")
    return _C.decode_cache(q, cache, scale, tau)
