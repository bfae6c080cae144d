"""The work that a user of this library has it do, as a list of cases that can be timed and compared.

Every case goes through the public entry points: the Python interface (`mlops_b200.attention`: encode, prefill, decode)
where it has the call, the C interface (include/mlops_fbla.h: qkv_at, decode_at, qkv_prefill_at, prefill_at -- device
lengths, per-row lengths) where an engine drives the library with positions that live on the GPU. The kinds:

  encode   quantise-on-write of dense K / V into a new cache
  prompt   an engine's prompt: norm + rotary embedding of the projection's rows, then causal prefill, count on the device
  prefill  causal attention of whole prompts, a batch of equal lengths
  chunk    one chunk of a long prompt behind a cached prefix
  verify   a few drafted tokens per sequence over a long cache (speculative decoding)
  decode   one token per sequence over the cache, equal lengths
  serving  one token per sequence, ragged per-row device lengths
  step     an engine's whole attention step: norm + rotary embedding + append of the new token, then the decode

Values: BF16 N(0, 1), 4 of the 128 channels of every (sequence, KV head) times 8 in K and V (the outlier channels of the
benchmark's configurations); head dimension 128 throughout.
"""
import ctypes

import torch

from mlops_b200 import attention
from mlops_b200.attention import _C

GROUP = 128
BITS = {"3+3": (3, 3), "4+2": (4, 2)}
TAU = {"3+3": 3e-4, "4+2": 1e-3}


def listed():
    return [
        # the smallest call: one sequence, a short context; launches and latency count
        dict(name="decode_4k", kind="decode", batch=1, q_heads=16, kv_heads=8, tokens=4096, mode="3+3"),
        # an engine's step at a small and at an ordinary batch, ragged lengths that are no multiples of anything
        dict(name="step_b1", kind="step", batch=1, q_heads=32, kv_heads=8, lo=1999, hi=1999, mode="4+2"),
        dict(name="step_b32", kind="step", batch=32, q_heads=32, kv_heads=8, lo=300, hi=6000, mode="3+3"),
        # the batched decode, the long context, the longest context of the benchmark's configurations
        dict(name="decode_b8_16k", kind="decode", batch=8, q_heads=32, kv_heads=8, tokens=16384, mode="4+2"),
        dict(name="decode_128k", kind="decode", batch=1, q_heads=32, kv_heads=8, tokens=131072, mode="3+3"),
        dict(name="decode_1m", kind="decode", batch=1, q_heads=32, kv_heads=8, tokens=1 << 20, mode="4+2"),
        # mixed serving: contexts of 1K to 64K tokens in one batch
        dict(name="serving_b64", kind="serving", batch=64, q_heads=32, kv_heads=8, lo=1024, hi=65536, mode="3+3"),
        # prompts: a short odd one, a batch of long ones, one chunk of a very long one
        dict(name="prompt_777", kind="prompt", q_heads=32, kv_heads=8, tokens=777, mode="3+3"),
        dict(name="prefill_b4_8k", kind="prefill", batch=4, q_heads=32, kv_heads=8, tokens=8192, mode="4+2"),
        dict(name="chunk_2k_at_64k", kind="chunk", batch=1, q_heads=16, kv_heads=8, tokens=2048, context=65536, mode="3+3"),
        # a handful of drafted tokens checked against a long context
        dict(name="verify_5_at_12k", kind="verify", batch=4, q_heads=32, kv_heads=8, tokens=5, context=12345, mode="4+2"),
        # a document's K / V written into a cache
        dict(name="encode_32k", kind="encode", batch=1, kv_heads=8, tokens=32768, mode="3+3"),
    ]


def _log(rng, lo, hi):
    """a whole number between lo and hi, spread over its logarithm"""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["decode", "decode", "step", "serving", "prompt", "prefill", "chunk", "verify", "encode"])
    kv_heads = rng.choice([2, 4, 8, 8])
    case = dict(kind=kind, q_heads=kv_heads * rng.choice([1, 2, 4, 4, 8 if kv_heads < 8 else 4]), kv_heads=kv_heads, mode=rng.choice(["3+3", "4+2"]))
    if kind == "decode":
        tokens = _log(rng, 200, 1 << 20)
        case.update(batch=_log(rng, 1, max(1, min(64, (1 << 20) // tokens))), tokens=tokens)
    elif kind == "serving":
        lo = _log(rng, 200, 4000)
        case.update(batch=_log(rng, 4, 64), lo=lo, hi=_log(rng, lo + 1000, 65536))
    elif kind == "step":
        lo = _log(rng, 200, 8000)
        case.update(batch=_log(rng, 1, 64), lo=lo, hi=_log(rng, lo, 8192))
    elif kind == "prompt":
        case.update(tokens=_log(rng, 90, 4096))
    elif kind == "prefill":
        batch = rng.randint(1, 4)
        case.update(batch=batch, tokens=_log(rng, 200, 8192))
    elif kind == "chunk":
        tokens = _log(rng, 200, 2048)
        case.update(batch=1, tokens=tokens, context=_log(rng, 2000, 65536 * 16 // max(16, case["q_heads"])))
    elif kind == "verify":
        case.update(batch=_log(rng, 1, 8), tokens=rng.randint(2, 8), context=_log(rng, 1000, 32768))
    else:
        del case["q_heads"]
        batch = _log(rng, 1, 8)
        case.update(batch=batch, tokens=_log(rng, 500, 131072 // batch))
    return case


# ---- inputs -----------------------------------------------------------------------------------------------------------------
def _normal(gen, *shape):
    return torch.randn(shape, generator=gen, dtype=torch.bfloat16, device="cuda")


def _kv(gen, batch, kv_heads, n, factors=None):
    """K and V [batch, kv_heads, n, 128]; `factors`: the outlier channels of the (sequence, head), the same for all its tokens"""
    if factors is None:
        factors = _factors(gen, batch, kv_heads)
    return _normal(gen, batch, kv_heads, n, 128).mul_(factors), _normal(gen, batch, kv_heads, n, 128).mul_(factors)


def _factors(gen, batch, kv_heads):
    order = torch.rand((batch, kv_heads, 1, 128), generator=gen, device="cuda").argsort(-1)
    return torch.where(order < 4, 8.0, 1.0).to(torch.bfloat16)


def _filled(gen, batch, kv_heads, tokens, mode, capacity):
    """a cache holding `tokens` tokens, written in pieces"""
    cache = attention.empty(batch, kv_heads, capacity, mode)
    factors = _factors(gen, batch, kv_heads)
    piece = max(1, (1 << 17) // batch)
    for t in range(0, tokens, piece):
        attention.append(cache, *_kv(gen, batch, kv_heads, min(piece, tokens - t), factors))
    return cache


def _lengths(gen, batch, lo, hi):
    n = torch.randint(lo, hi + 1, (batch,), generator=gen, device="cuda", dtype=torch.int32)
    # no token of these passes opens a group (1 step in 128 does): a pass can then be repeated on the same cache
    return torch.where(n % GROUP == 0, n - 1, n).to(torch.int32)


def _ragged(gen, batch, kv_heads, lengths, mode, capacity):
    """one cache whose row b holds lengths[b] tokens"""
    cache = attention.empty(batch, kv_heads, capacity, mode)
    arrays = ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v")
    for b, n in enumerate(lengths.tolist()):
        row = attention.FBLACache(**{a: getattr(cache, a)[b:b + 1] for a in arrays}, tokens=0, capacity=capacity, format=cache.format)
        attention.append(row, *_kv(gen, 1, kv_heads, n))
    return cache


class _Token(ctypes.Structure):
    """mlops_fbla_token"""
    _fields_ = [("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("v", ctypes.c_void_p), ("batch_stride", ctypes.c_int64),
                ("q_group_stride", ctypes.c_int64), ("kv_group_stride", ctypes.c_int64), ("q_norm", ctypes.c_void_p), ("k_norm", ctypes.c_void_p),
                ("eps", ctypes.c_float), ("freq", ctypes.c_void_p), ("attention_factor", ctypes.c_float), ("q_out", ctypes.c_void_p)]


def _frequencies(theta=1e6):
    """the rotary table of mlops_fbla_token: per pair f = inv_freq / 2 pi and frac(65536 f), each as a float and its remainder"""
    f = theta ** (-torch.arange(0, 128, 2, dtype=torch.float64) / 128) / (2 * torch.pi)
    g = (65536 * f) % 1.0
    hi = lambda x: x.to(torch.float32)  # noqa: E731
    lo = lambda x: (x - x.to(torch.float32).to(torch.float64)).to(torch.float32)  # noqa: E731
    return torch.stack([hi(f), lo(f), hi(g), lo(g)], dim=1).contiguous().cuda()


def _token(s, proj, q_heads, kv_heads, q_out):
    """rows of the projection: per KV head its q heads, then k, then v"""
    qg = q_heads // kv_heads
    base, row = proj.data_ptr(), kv_heads * (qg + 2) * 128
    return _Token(base, base + 2 * qg * 128, base + 2 * (qg + 1) * 128, row, (qg + 2) * 128, (qg + 2) * 128, s["q_norm"].data_ptr(),
                  s["k_norm"].data_ptr(), 1e-6, s["freq"].data_ptr(), 0.0, q_out.data_ptr() if q_out is not None else None)


def _struct(c):
    return _C.Cache(c.coarse.data_ptr(), c.fine.data_ptr(), c.meta.data_ptr(), c.sink_k.data_ptr(), c.sink_v.data_ptr(), c.open_k.data_ptr(),
                    c.open_v.data_ptr(), None)


def _check(status):
    if status:
        raise RuntimeError(_C.last_error())


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, kv_heads, mode = case["kind"], case["kv_heads"], case["mode"]
    batch, q_heads = case.get("batch", 1), case.get("q_heads", 0)
    s = dict(kind=kind, mode=mode)
    if kind == "encode":
        s["k"], s["v"] = _kv(gen, batch, kv_heads, case["tokens"])
    elif kind == "decode":
        s["cache"] = _filled(gen, batch, kv_heads, case["tokens"], mode, case["tokens"])
        s["q"] = _normal(gen, batch, q_heads, 128)
    elif kind in ("prefill", "chunk", "verify"):
        n, n0 = case["tokens"], case.get("context", 0)
        if kind == "verify":  # the drafted tokens stay inside the open group: what a later pass finds there is what this one found
            n0 = n0 // GROUP * GROUP + min(max(n0 % GROUP, 1), GROUP - n)
        s["cache"] = _filled(gen, batch, kv_heads, n0, mode, n0 + n)
        s["held"] = n0
        s["k"], s["v"] = _kv(gen, batch, kv_heads, n)
        s["q"] = _normal(gen, batch, q_heads, n, 128)
        if kind == "chunk":
            s["open"] = s["cache"].open_k.clone(), s["cache"].open_v.clone()
    else:
        s["q_norm"], s["k_norm"] = (1 + 0.1 * _normal(gen, 128)), (1 + 0.1 * _normal(gen, 128))
        s["freq"] = _frequencies()
        row = kv_heads * (q_heads // kv_heads + 2) * 128
        if kind == "prompt":
            n = case["tokens"]
            ceiling = -(-n // 256) * 256  # an engine pads its chunk buffers; the count lives on the device
            s["cache"] = attention.empty(1, kv_heads, ceiling, mode)
            s["proj"] = _normal(gen, n, row)
            s["length"], s["count"] = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.full((1,), n, dtype=torch.int32, device="cuda")
            s["q"], s["out"] = (torch.zeros((q_heads, ceiling, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
            s["k"], s["v"] = (torch.zeros((kv_heads, ceiling, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
            s["n"], s["ceiling"] = n, ceiling
            s["token"] = _token(s, s["proj"], q_heads, kv_heads, None)
            s["config"] = _C.Config(1, q_heads, kv_heads, 0, 0.0, 0.0, s["cache"].format, ceiling, 0, 0, 0, 0, 0)
        else:
            s["length"] = _lengths(gen, batch, case["lo"], case["hi"])
            capacity = -(-(case["hi"] + 1) // 256) * 256  # whole pages of 256 tokens
            s["cache"] = _ragged(gen, batch, kv_heads, s["length"], mode, capacity)
            sized = _C.Config(batch, q_heads, kv_heads, capacity, 0.0, 0.0, s["cache"].format, capacity, 0, 0, 0, 0, 0)
            s["scratch"] = torch.empty(_C.lib.mlops_fbla_decode_scratch_bytes(ctypes.byref(sized)), dtype=torch.uint8, device="cuda")
            s["q"] = _normal(gen, batch, q_heads, 128)
            s["out"] = torch.zeros_like(s["q"])
            # the decode of a step counts the token that the step appended
            s["config"] = _C.Config(batch, q_heads, kv_heads, 1 if kind == "step" else 0, 0.0, 0.0, s["cache"].format, capacity, 0, 0, 0, 0, 1)
            if kind == "step":
                s["proj"] = _normal(gen, batch, row)
                s["token"] = _token(s, s["proj"], q_heads, kv_heads, s["q"])
                s["append"] = _C.Config(batch, q_heads, kv_heads, 0, 0.0, 0.0, s["cache"].format, capacity, 0, 0, 0, 0, 1)
        s["struct"] = _struct(s["cache"])
    return s


def _written(c):
    return dict(coarse=c.coarse, fine=c.fine, meta=c.meta, sink_k=c.sink_k, sink_v=c.sink_v, open_k=c.open_k, open_v=c.open_v)


def run(s):
    kind = s["kind"]
    if kind == "encode":
        return _written(attention.encode(s["k"], s["v"], s["mode"]))
    if kind == "decode":
        return attention.decode(s["q"], s["cache"])
    if kind in ("prefill", "chunk", "verify"):
        cache = s["cache"]
        cache.tokens = s["held"]  # a reused slot; a request that branches off a shared prefix; rejected drafts dropped
        if kind == "chunk":
            cache.open_k.copy_(s["open"][0])
            cache.open_v.copy_(s["open"][1])
        out = attention.prefill(s["q"], s["k"], s["v"], cache)
        return dict(out=out, open_k=cache.open_k, open_v=cache.open_v) if kind == "verify" else dict(out=out, **_written(cache))
    lib, ref, ptr = _C.lib, ctypes.byref, lambda t: ctypes.c_void_p(t.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "prompt":
        _check(lib.mlops_fbla_qkv_prefill_at(ref(s["config"]), ptr(s["length"]), ptr(s["count"]), s["ceiling"], ref(s["token"]), ptr(s["q"]), ptr(s["k"]),
                                             ptr(s["v"]), stream))
        _check(lib.mlops_fbla_prefill_at(ref(s["config"]), ptr(s["length"]), ptr(s["count"]), s["ceiling"], ptr(s["q"]), ptr(s["k"]), ptr(s["v"]),
                                         ref(s["struct"]), ptr(s["out"]), stream))
        return dict(q=s["q"], k=s["k"], v=s["v"], out=s["out"][:, :s["n"]], **_written(s["cache"]))
    if kind == "step":
        _check(lib.mlops_fbla_qkv_at(ref(s["append"]), ptr(s["length"]), ref(s["token"]), ref(s["struct"]), stream))
    _check(lib.mlops_fbla_decode_at(ref(s["config"]), ptr(s["length"]), ptr(s["q"]), ref(s["struct"]), ptr(s["out"]), ptr(s["scratch"]),
                                    s["scratch"].numel(), stream))
    if kind == "step":
        return dict(q=s["q"], out=s["out"], open_k=s["cache"].open_k, open_v=s["cache"].open_v)
    return s["out"]


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------
def _decode_work(batch, q_heads, kv_heads, tokens, mode):
    """The coarse records and metadata of the closed groups, the BF16 windows, q and the output; the fine records where the
    average 16-token block holds more of a query's softmax mass than tau (values like these spread it evenly)."""
    cb, fb = BITS[mode]
    closed = max((tokens + GROUP - 1) // GROUP - 2, 0)
    unit = 8 * 512 * cb + 1024 + (8 * 512 * fb if 16 / tokens > TAU[mode] else 0)
    window = min(tokens, GROUP) + (tokens - GROUP * (closed + 1) if tokens > GROUP else 0)
    return batch * (kv_heads * (closed * unit + window * 512) + 2 * q_heads * 256), 4 * 128 * batch * q_heads * tokens


def _chunk_work(batch, q_heads, kv_heads, context, n):
    """q, k, v and the output of the chunk, the cache behind it, the groups that it closes; four products' operations per
    attended (query, key) pair and channel"""
    data = batch * n * 256 * (2 * q_heads + 2 * kv_heads) + batch * kv_heads * (context + n) * 200
    return data, 4 * 128 * batch * q_heads * (n * context + n * (n + 1) // 2)


def work(case):
    kind, kv_heads = case["kind"], case["kv_heads"]
    batch, q_heads = case.get("batch", 1), case.get("q_heads", 0)
    if kind == "encode":
        n = batch * kv_heads * case["tokens"]
        return {"bytes": n * 512 + n * 200, "flops": 0}
    if kind == "decode":
        data, flops = _decode_work(batch, q_heads, kv_heads, case["tokens"], case["mode"])
    elif kind in ("serving", "step"):  # evenly spread lengths: eight of them stand for all
        steps = [case["lo"] + (case["hi"] - case["lo"]) * (2 * i + 1) // 16 for i in range(8)]
        parts = [_decode_work(1, q_heads, kv_heads, n, case["mode"]) for n in steps]
        data, flops = (batch * sum(p[i] for p in parts) // 8 for i in (0, 1))
        if kind == "step":
            data += batch * (q_heads + 2 * kv_heads) * 512
    else:
        n = case["tokens"]
        data, flops = _chunk_work(batch, q_heads, kv_heads, case.get("context", 0), n)
        if kind == "prompt":
            data += n * (q_heads + 2 * kv_heads) * 512
    return {"bytes": data, "flops": flops}


def tolerance(case):
    """Cache bytes are whole numbers and stay the same. Attention outputs are BF16, of 8-bit softmax weights and 6-bit codes:
    two correct implementations differ by the rounding of the output and by weights that round the other way."""
    return "exact" if case["kind"] == "encode" else {"rel": 1e-2, "max": 0.1}
