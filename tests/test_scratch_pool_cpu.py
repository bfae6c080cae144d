"""The Python decode's pool of scratch buffers, without a GPU: one buffer per stream, grown on demand, a bounded number."""
import os

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def pool_type():
    if not os.path.exists(os.path.join(ROOT, "mlops_b200", "lib", "libmlops_attention.so")):
        import __graft_entry__
        __graft_entry__.build()
    from mlops_b200.attention import _C
    return _C._ScratchPool


def test_one_buffer_per_stream_and_a_bounded_number(pool_type):
    pool, cpu = pool_type(), torch.device("cpu")
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
