"""The few-row prefill attention (chunks of fewer than 64 rows per KV head) where its dealing can go wrong: no cache, one
group, a chunk that crosses a group boundary, tiles with padding rows, one and several shares of a tile's groups, several
tiles to a CTA (the last CTA's fewer); host and device lengths and an executor's items bit for bit."""
import ctypes

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
@pytest.mark.parametrize("B,QH,KH,n0,n", [(1, 1, 1, 0, 1), (1, 4, 2, 0, 20), (2, 2, 2, 127, 3), (1, 8, 2, 250, 13), (3, 4, 1, 1000, 5), (1, 2, 1, 128, 31),
                                          (1, 8, 2, 5000, 6), (1, 1, 1, 9215, 2), (4, 16, 4, 3000, 1), (1, 6, 2, 12345, 21),
                                          (4, 8, 8, 1669, 36), (1, 8, 8, 6275, 43), (4, 24, 24, 2000, 25)])
def test_few_rows(ours, oracle, mode, B, QH, KH, n0, n):
    q, k, v = datagen.uneven_case(n0 + n, B, QH, KH, n0 + n, q_rows=n0 + n)
    q = q[:, :, n0:].copy()
    cap = n0 + n + 9
    o = oracle.empty(B, KH, cap, mode)
    c = ours.empty(B, KH, cap, mode)
    if n0:
        oracle.append(o, k[:, :, :n0], v[:, :, :n0])
        ours.prefill(c, gu.bf16_tensor(k[:, :, :n0]), gu.bf16_tensor(v[:, :, :n0]))
    start = {key: (val.clone() if torch.is_tensor(val) else val) for key, val in c.items()}
    qd, kd, vd = gu.bf16_tensor(q), gu.bf16_tensor(k[:, :, n0:]), gu.bf16_tensor(v[:, :, n0:])
    got = ours.prefill(c, kd, vd, qd)
    torch.cuda.synchronize()
    gu.check_close(gu.bits_of(got), oracle.prefill(q, k[:, :, n0:], v[:, :, n0:], o), f"{mode} {n} rows at {n0}")
    gu.assert_cache_equal(c, o, mode)
    # the same chunk with its start and count on the device
    length, count = (torch.tensor([x], dtype=torch.int32, device="cuda") for x in (n0, n))
    d = {key: (val.clone() if torch.is_tensor(val) else val) for key, val in start.items()}
    out = torch.full_like(got, -7.0)
    ours.prefill_at(d, kd, vd, qd, length, count, n, out=out)
    torch.cuda.synchronize()
    assert torch.equal(out, got)
    # and as an executor's items, which take a tile's shares one after the other
    kc = ours._cache(start)
    cfg = gu.Config(B, QH, KH, 0, 0, 0, gu.FORMATS[mode][2], cap, 0, 0, 0, 0, 0)
    out = torch.full_like(got, -7.0)
    passes, vp = (iu.Items * 4)(), ctypes.c_void_p
    npass = ours.lib.mlops_fbla_prefill_at_items(ctypes.byref(cfg), vp(length.data_ptr()), vp(count.data_ptr()), n, vp(qd.data_ptr()), vp(kd.data_ptr()),
                                                 vp(vd.data_ptr()), ctypes.byref(kc), vp(out.data_ptr()), passes, 4)
    assert npass == 3, ours.error()
    iu.run_plan(ours.lib, passes, npass, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(out, got)
