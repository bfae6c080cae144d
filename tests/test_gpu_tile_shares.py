"""The tensor-core prefill with a tile's passes split over a cluster: shares that begin and end among closed and BF16 groups, a
share without passes, a last tile with few rows, ragged ends; against the oracle, and host against device lengths."""
import numpy as np
import pytest
import torch

from tests import datagen
from tests import gpu_util as gu

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
