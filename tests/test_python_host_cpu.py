"""The Python side without a GPU: the decode's pool of scratch buffers (one per stream, grown on demand, a bounded number) and the tensors of
a cache record."""
import os

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def package():
    if not os.path.exists(os.path.join(ROOT, "mlops_b200", "lib", "libmlops_attention.so")):
        import __graft_entry__
        __graft_entry__.build()
    from mlops_b200 import attention
    return attention


def test_one_buffer_per_stream_and_a_bounded_number(package):
    pool, cpu = package._C._ScratchPool(), torch.device("cpu")
    first = pool.get(cpu, 1, 1000)
    assert pool.get(cpu, 1, 10) is first and pool.get(cpu, 1, 1000) is first and first.buffer.numel() == 1000
    grown = pool.get(cpu, 1, 1001)
    assert grown is not first and grown.bytes == 1001 and pool.get(cpu, 1, 5) is grown
    assert pool.get(cpu, 2, 5) is not grown
    for stream in range(3, 3 + pool.BUFFERS):
        pool.get(cpu, 1, 5)  # (in use: stays)
        pool.get(cpu, stream, 5)
    assert len(pool._held) == pool.BUFFERS and pool.get(cpu, 1, 5) is grown
    assert not first.lock.locked() and first.lock is not grown.lock


def test_the_arrays_of_a_cache_are_tensors_of_their_own(package):
    """Each can be written, saved and given back without the others (a window that was a view of all four could not be written while autograd
    records)."""
    cache = package.fbla._allocate(torch.zeros, torch.zeros_like, 1, 2, 300, "4+2", "cpu")
    arrays = [cache.coarse, cache.fine, cache.meta, cache.sink_k, cache.sink_v, cache.open_k, cache.open_v]
    assert len({a.untyped_storage().data_ptr() for a in arrays}) == 7
    assert all(a.untyped_storage().nbytes() == a.numel() * a.element_size() for a in arrays)
    cache.open_k.copy_(torch.ones_like(cache.open_k, requires_grad=True))
    assert cache.open_k.requires_grad and not cache.open_v.requires_grad
