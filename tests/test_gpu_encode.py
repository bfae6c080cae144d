"""mlops_fbla_encode into arrays without initial contents gives the bytes of a zeroed cache and an append: lengths around
the group boundary, capacities beyond the tokens, both formats."""
import ctypes

import pytest
import torch

from mlops_b200 import attention
from mlops_b200.attention import _C

pytestmark = pytest.mark.gpu
ARRAYS = ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v")


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("n,capacity", [(1, 1), (5, 700), (127, 127), (128, 128), (129, 129), (129, 1000), (300, 384), (1025, 4096)])
def test_encode_needs_no_initial_contents(mode, n, capacity):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    k, v = (torch.randn((2, 3, n, 128), generator=gen, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    want = attention.append(attention.empty(2, 3, capacity, mode), k, v)
    got = attention.empty(2, 3, capacity, mode)
    for a in ARRAYS:
        getattr(got, a).view(torch.uint8).fill_(0xA5)
    _C.encode(k, v, *[getattr(got, a) for a in ARRAYS], capacity, got.format)
    whole = attention.encode(k, v, mode, capacity)
    for a in ARRAYS:
        x = getattr(want, a).view(torch.uint8)
        assert torch.equal(getattr(got, a).view(torch.uint8), x), a
        assert torch.equal(getattr(whole, a).view(torch.uint8), x), a
    assert whole.tokens == want.tokens == n


def test_encode_starts_an_empty_cache_only():
    c = attention.empty(1, 1, 256)
    kc = _C._cache(*[getattr(c, a) for a in ARRAYS])
    cfg = _C._config(1, 1, 1, 5, 0, 256, 0.0, 0.0)
    assert _C.lib.mlops_fbla_encode(ctypes.byref(cfg), 1, c.open_k.data_ptr(), c.open_v.data_ptr(), ctypes.byref(kc), None) == _C.INVALID_VALUE
    assert "tokens has to be 0" in _C.last_error()


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("heads,n,n0", [(8, 12300, 0), (3, 40001, 0), (5, 9000, 77)])
def test_many_units_per_cta(oracle, mode, heads, n, n0):
    """More (group, tensor) units than CTAs: the later ones come through shared memory; a chunk that starts inside a group; channels whose
    steps are subnormal, have a subnormal reciprocal, or none (a constant channel, a range beyond the largest float) beside ordinary ones."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    scale = 2.0 ** torch.randint(-12, 3, (1, heads, 1, 128), generator=gen, device="cuda").double()
    scale[..., 3], scale[..., 50], scale[..., 90], scale[..., 127] = 2.0 ** -131, 2.0 ** -124, 2.0 ** 124, 2.0 ** 127
    k, v = ((torch.randn((1, heads, n0 + n, 128), generator=gen, device="cuda").clamp(-1.9, 1.9).double() * scale).to(torch.bfloat16) for _ in range(2))
    k[..., 17], v[..., 18] = 0.5, 0.0
    c = attention.empty(1, heads, n0 + n + 300, mode)
    if n0:
        attention.append(c, k[:, :, :n0], v[:, :, :n0])
    attention.append(c, k[:, :, n0:], v[:, :, n0:])
    bits = lambda x: x.view(torch.int16).cpu().numpy().view("uint16")  # noqa: E731
    want = oracle.encode(bits(k), bits(v), mode, capacity=n0 + n + 300)
    for a in ARRAYS:
        x, y = getattr(c, a).view(torch.uint8).cpu().numpy().reshape(-1), want[a].view("uint8").reshape(-1)
        assert x.size == y.size and (x == y).all(), a


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
def test_values_that_are_not_numbers_or_infinite(oracle, mode):
    """Records and metadata byte for byte the oracle's where channels hold NaN (code 0, not part of the range) and infinities (no step: code 0)"""
    heads, n = 8, 12300
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    k, v = (torch.randn((1, heads, n, 128), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    for x in (k, v):
        rare = torch.rand((1, heads, n), generator=gen, device="cuda") < 0.03
        x[..., 5] = torch.where(rare, float("nan"), x[..., 5])
        x[..., 70] = torch.where(rare, float("inf"), x[..., 70])
        x[..., 99] = torch.where(rare, float("-inf"), x[..., 99])
        x[..., 100] = torch.where(rare, float("nan"), x[..., 99])
        x[:, :, 256:384, 31] = float("nan")
        x[:, :, 256:384, 32] = float("-inf")
    c = attention.empty(1, heads, n, mode)
    attention.append(c, k, v)
    bits = lambda x: x.view(torch.int16).cpu().numpy().view("uint16")  # noqa: E731
    want = oracle.encode(bits(k), bits(v), mode)
    for a in ARRAYS:
        x, y = getattr(c, a).view(torch.uint8).cpu().numpy().reshape(-1), want[a].view("uint8").reshape(-1)
        assert x.size == y.size and (x == y).all(), a
