"""The Python cache record and what the calls on it keep: a cache that has been in use can be copied, pickled and saved; every call
looks at the arrays it is given; the decode's scratch is nobody else's (threads on one stream, captured graphs)."""
import copy
import io
import pickle
import threading

import pytest
import torch

from mlops_b200 import attention

pytestmark = pytest.mark.gpu
ARRAYS = ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v")


def _case(tokens=300, batch=1, q_heads=4, kv_heads=2, mode="3+3", capacity=1024):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(tokens)
    k, v = (torch.randn((batch, kv_heads, tokens, 128), generator=gen, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    return torch.randn((batch, q_heads, 128), generator=gen, dtype=torch.bfloat16, device="cuda"), attention.encode(k, v, mode, capacity)


def _saved(cache):
    file = io.BytesIO()
    torch.save(cache, file)
    file.seek(0)
    return torch.load(file, weights_only=False)


@pytest.mark.parametrize("branch", [copy.deepcopy, lambda c: pickle.loads(pickle.dumps(c)), _saved], ids=["deepcopy", "pickle", "save"])
def test_a_cache_in_use_can_be_branched(branch):
    q, cache = _case()
    want = attention.decode(q, cache)
    attention.append(cache, *(torch.zeros((1, 2, 1, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2)))
    other = branch(cache)
    assert other.tokens == cache.tokens == 301
    for a in ARRAYS:
        assert torch.equal(getattr(other, a), getattr(cache, a)) and getattr(other, a).data_ptr() != getattr(cache, a).data_ptr()
    kept = other.open_k.clone()
    attention.append(cache, *(torch.ones((1, 2, 1, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2)))
    assert torch.equal(other.open_k, kept)
    other.tokens = 300
    assert torch.equal(attention.decode(q, other), want)


def test_every_call_looks_at_the_arrays():
    q, cache = _case()
    attention.decode(q, cache)
    cache.open_k.transpose_(2, 3)  # (the same tensor at the same address, no longer the layout the library reads)
    with pytest.raises(ValueError, match="contiguous"):
        attention.decode(q, cache)
    cache.open_k.transpose_(2, 3)
    attention.decode(q, cache)
    cache.sink_v.transpose_(2, 3)
    with pytest.raises(ValueError, match="contiguous"):
        attention.append(cache, *(torch.zeros((1, 2, 1, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2)))


def test_a_captured_decode_keeps_its_scratch():
    """A graph's kernels name the scratch of the calls it was captured from: nothing that runs later may be given that memory, however
    many streams decode in between."""
    q, cache = _case(3000, 2, 8, 2, capacity=4096)
    want = attention.decode(q, cache)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        attention.decode(q, cache)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = attention.decode(q, cache)
    others = [torch.cuda.Stream() for _ in range(20)]
    for s in others:
        with torch.cuda.stream(s):
            attention.decode(q, cache)
    torch.cuda.synchronize()
    nbytes = attention._C.scratch_bytes(2, 8, 2, 4096, cache.format, 4096)
    with torch.cuda.stream(stream):
        guards = [torch.full((nbytes,), 0x5A, dtype=torch.uint8, device="cuda") for _ in range(4)]
    stream.synchronize()
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert all(bool((g == 0x5A).all()) for g in guards)


def test_threads_on_one_stream():
    """Two threads that decode on the same stream share its scratch: the kernels of one call are never enqueued between another's."""
    cases = [_case(n, 1, 8, 2, capacity=4096) for n in (3001, 3002)]
    want = [attention.decode(*c) for c in cases]
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(2)

    def work(i):
        start.wait()
        outs = [attention.decode(*cases[i]) for _ in range(300)]
        torch.cuda.synchronize()
        wrong.extend(k for k, o in enumerate(outs) if not torch.equal(o, want[i]))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_scratch_follows_the_tokens():
    """A slot with room for more tokens than one decode takes is decoded as long as it holds no more than that."""
    q, cache = _case(300)
    slot = attention.empty(1, 2, (1 << 26) + 128, "3+3")
    for a in ARRAYS:
        held = getattr(cache, a)
        getattr(slot, a)[:, :, :held.shape[2]].copy_(held)
    slot.tokens = 300
    got, want = (attention.decode(q, c).float() for c in (slot, cache))
    assert float((got - want).abs().max()) <= 2e-3 * float(want.abs().max()) + 2.0 ** -7 * float(want.abs().max())
