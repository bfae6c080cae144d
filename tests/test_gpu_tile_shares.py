"""The tensor-core prefill with a tile's passes split over a cluster: shares that begin and end among closed and BF16 groups, a
share without passes, a last tile with few rows, ragged ends; against the oracle, and host against device lengths."""
import ctypes

import numpy as np
import pytest
import torch

from tests import datagen
from tests import gpu_util as gu
from tests import items_util as iu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ours():
    return gu.CLib(gu.OURS)


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("B,QH,KH,n0,n,step", [(1, 1, 1, 9000, 64, 7), (1, 2, 1, 0, 3200, 61), (2, 4, 2, 4999, 130, 9), (1, 8, 1, 12801, 77, 5), (1, 2, 2, 3071, 257, 16)])
def test_split_passes(ours, oracle, mode, B, QH, KH, n0, n, step):
    q, k, v = datagen.uneven_case(n0 + n, B, QH, KH, n0 + n, q_rows=n0 + n)
    q = q[:, :, n0:].copy()
    cap = n0 + n
    o, c = oracle.empty(B, KH, cap, mode), ours.empty(B, KH, cap, mode)
    if n0:
        oracle.append(o, k[:, :, :n0], v[:, :, :n0])
        ours.prefill(c, gu.bf16_tensor(k[:, :, :n0]), gu.bf16_tensor(v[:, :, :n0]))
    d = {key: (val.clone() if torch.is_tensor(val) else val) for key, val in c.items()}
    qd, kd, vd = gu.bf16_tensor(q), gu.bf16_tensor(k[:, :, n0:]), gu.bf16_tensor(v[:, :, n0:])
    got = ours.prefill(c, kd, vd, qd)
    torch.cuda.synchronize()
    at = np.arange(0, n, step)
    want = oracle.prefill(q, k[:, :, n0:], v[:, :, n0:], o, pos_step=step)
    gu.check_close(gu.bits_of(got)[:, :, at], want[:, :, at], f"{mode} {n} at {n0}")
    gu.assert_cache_equal(c, o, mode)
    length, count = (torch.tensor([x], dtype=torch.int32, device="cuda") for x in (n0, n))
    out = torch.full_like(got, -7.0)
    ours.prefill_at(d, kd, vd, qd, length, count, n, out=out)
    torch.cuda.synchronize()
    assert torch.equal(out, got)
    d["tokens"] = c["tokens"]
    gu.assert_cache_equal(d, o, f"{mode}, device length")


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("QH,KH,n0,n,cap", [(8, 2, 12001, 77, 16384), (8, 2, 700, 130, 16384), (4, 2, 9000, 700, 16384), (2, 1, 6000, 1500, 8192)])
def test_same_bits_for_every_ceiling_and_for_items(ours, mode, QH, KH, n0, n, cap):
    """How a tile's passes are shared out follows from the chunk's own size: the call with the count on the host, with the count on the
    device under any ceiling (one launch or two, the shares of the ceiling's size fewer than, or the same as, the chunk's), and the plan's
    items, which take the shares in turn, give the same bits."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n0 + n)
    normal = lambda *shape: torch.randn(shape, generator=gen, dtype=torch.bfloat16, device="cuda")  # noqa: E731
    base = ours.empty(1, KH, cap, mode)
    ours.prefill(base, normal(1, KH, n0, 128), normal(1, KH, n0, 128))
    copy = lambda: {key: (val.clone() if torch.is_tensor(val) else val) for key, val in base.items()}  # noqa: E731
    q, k, v = normal(1, QH, n, 128), normal(1, KH, n, 128), normal(1, KH, n, 128)
    want = ours.prefill(copy(), k, v, q)
    length, count = (torch.tensor([x], dtype=torch.int32, device="cuda") for x in (n0, n))
    pad = lambda x, m: torch.nn.functional.pad(x, (0, 0, 0, m - n)).contiguous()  # noqa: E731
    for ceiling in sorted({n, n + 1, min(2 * n, cap - n0), min(8 * n, cap - n0), cap - n0}):
        out = torch.full((1, QH, ceiling, 128), -7.0, dtype=torch.bfloat16, device="cuda")
        ours.prefill_at(copy(), pad(k, ceiling), pad(v, ceiling), pad(q, ceiling), length, count, ceiling, out=out)
        assert torch.equal(out[:, :, :n], want), ceiling
        assert (out[:, :, n:] == -7.0).all()
    pytest.importorskip("cuda.bindings.nvrtc")
    lib, vp, ceiling, c = ours.lib, ctypes.c_void_p, min(2 * n, cap - n0), copy()
    out = torch.full((1, QH, ceiling, 128), -7.0, dtype=torch.bfloat16, device="cuda")
    cfg = gu.Config(1, QH, KH, 0, 0, 0, gu.FORMATS[mode][2], cap, 0, 0, 0, 0, 0)
    passes, kc, padded = (iu.Items * 4)(), ours._cache(c), [pad(x, ceiling) for x in (q, k, v)]
    got = lib.mlops_fbla_prefill_at_items(ctypes.byref(cfg), vp(length.data_ptr()), vp(count.data_ptr()), ceiling, *(vp(x.data_ptr()) for x in padded),
                                          ctypes.byref(kc), vp(out.data_ptr()), passes, 4)
    assert got > 0, ours.error()
    iu.run_plan(lib, passes, got, torch.cuda.current_stream().cuda_stream, 3)
    assert torch.equal(out[:, :, :n], want)
    assert (out[:, :, n:] == -7.0).all()
