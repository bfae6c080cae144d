"""The dense decode (scores first, then every sub-block's value once) and the decode that corrects coarse sums, at the
lengths where dealing or table look-ups can go wrong, against the oracle: no closed group, one, runs that end inside a
group; 1, 2 and 4 queries per virtual head; ragged rows; selection of none, some and all sub-blocks; shards of such rows."""
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
@pytest.mark.parametrize("B,QH,KH,N,tau", [(1, 1, 1, 1, 0.0), (1, 4, 1, 128, 0.0), (2, 8, 2, 256, 1e-6), (1, 2, 1, 257, 0.0), (1, 2, 2, 385, 2e-2),
                                           (3, 8, 2, 1025, 4e-3), (1, 24, 2, 700, 1e-3), (17, 4, 1, 3000, 0.0), (2, 16, 8, 9001, 1e-3), (1, 1, 1, 20011, 1e-9)])
def test_dense_sizes(ours, oracle, mode, B, QH, KH, N, tau):
    q, k, v = datagen.baseline_case(7 + N, B, QH, KH, N)
    c = ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode)
    got = ours.decode(c, gu.bf16_tensor(q), tau=tau)
    again = ours.decode(c, gu.bf16_tensor(q), tau=tau)
    torch.cuda.synchronize()
    assert torch.equal(got, again)
    gu.check_close(gu.bits_of(got), oracle.decode(q, oracle.encode(k, v, mode), tau=tau), f"{mode} {N}")


@pytest.mark.parametrize("B,QH,KH,N", [(64, 32, 8, 300), (70, 16, 8, 700), (100, 8, 8, 390), (148, 16, 4, 513)])
def test_heads_folded_inside_a_cta(ours, oracle, B, QH, KH, N):
    """several heads per CTA, each of several warps, of one, and across the CTA's border"""
    q, k, v = datagen.baseline_case(5 + N, B, QH, KH, N)
    for mode in ("3+3", "4+2"):
        got = ours.decode(ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode), gu.bf16_tensor(q))
        torch.cuda.synchronize()
        gu.check_close(gu.bits_of(got), oracle.decode(q, oracle.encode(k, v, mode)), f"{mode} {B} x {N}")


# a cluster of 16, 10, 8, 6, 5, 4, 3, 2, 1 CTAs per head; CTAs without groups, without windows, with less and with more than a unit per warp
OWN = [(1, 4, 1, 130, 16), (1, 2, 1, 385, 16), (2, 3, 3, 9000, 16), (2, 16, 4, 2600, 10), (3, 8, 4, 3001, 8), (3, 24, 6, 257, 6), (5, 10, 5, 2999, 5), (8, 16, 4, 1700, 4),
       (9, 4, 4, 2049, 3), (9, 32, 4, 1500, 2), (16, 32, 8, 640, 1), (30, 8, 4, 2300, 1), (74, 4, 2, 17, 1)]


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("B,QH,KH,N,ctas", OWN)
def test_heads_with_ctas_of_their_own(ours, oracle, mode, B, QH, KH, N, ctas):
    q, k, v = datagen.baseline_case(11 + N, B, QH, KH, N)
    qd = gu.bf16_tensor(q)
    c = ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode, capacity=N)
    got = ours.decode(c, qd)
    assert torch.equal(got, ours.decode_at(c, qd, torch.tensor([N], dtype=torch.int32, device="cuda")))
    torch.cuda.synchronize()
    gu.check_close(gu.bits_of(got), oracle.decode(q, oracle.encode(k, v, mode, capacity=N)), f"{mode} {B} x {N}")
    assert ours.lib.fbla_k_head_ctas(B * KH * (QH // KH // gu_group(QH // KH)), ctypes.c_longlong(N)) == ctas
    assert first_entry(ours, c, qd, mode, 0.0).endswith(", true>")


def gu_group(ratio):
    """queries per virtual head"""
    return ratio if ratio in (1, 2, 4) else 4 if ratio % 4 == 0 else 2 if ratio % 2 == 0 else 1


@pytest.mark.parametrize("B,QH,KH,N,ctas", [OWN[2], OWN[3], OWN[5], OWN[10]])
def test_own_ctas_lengths_and_plans(ours, oracle, B, QH, KH, N, ctas):
    """Rows shorter than the room (down to one token, no closed group), each against its own decode in a cache of the same room; the plan's
    passes bit for bit the stream call, one CTA per item and as loops of three."""
    mode, lens = "4+2", [max(1, N * i // B - 3 * i) for i in range(B)]
    q, k, v = datagen.uneven_case(21, B, QH, KH, N)
    qd = gu.bf16_tensor(q)
    c = ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode, capacity=N)
    want = []
    for b, n in enumerate(lens):
        row = ours.encode(gu.bf16_tensor(k[b:b + 1, :, :n]), gu.bf16_tensor(v[b:b + 1, :, :n]), mode, capacity=N)
        for key in ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v"):
            c[key][b].copy_(row[key][0])
        want.append(oracle.decode(q[b:b + 1], oracle.encode(k[b:b + 1, :, :n], v[b:b + 1, :, :n], mode, capacity=N)))
    length, vp, passes = torch.tensor(lens, dtype=torch.int32, device="cuda"), ctypes.c_void_p, (iu.Items * 4)()
    got = ours.decode_at(c, qd, length, length_stride=1)
    torch.cuda.synchronize()
    for b in range(B):
        gu.check_close(gu.bits_of(got)[b:b + 1], want[b], f"row of {lens[b]}")
    cfg, kc = gu.Config(B, QH, KH, 0, 0, 0, gu.FORMATS[mode][2], N, 0, 0, 0, 0, 1), ours._cache(c)
    for loops in (None, 3):
        scratch, out = ours.scratch(dict(c, tokens=N), QH), torch.empty_like(qd)
        scratch.fill_(0xFF)
        assert ours.lib.mlops_fbla_decode_at_items(ctypes.byref(cfg), vp(length.data_ptr()), vp(qd.data_ptr()), ctypes.byref(kc), vp(out.data_ptr()),
                                                   vp(scratch.data_ptr()), ctypes.c_size_t(scratch.numel()), 0, passes, 4) == 4, ours.error()
        iu.run_plan(ours.lib, passes, 4, torch.cuda.current_stream().cuda_stream, loops)
        torch.cuda.synchronize()
        assert torch.equal(out, got)


@pytest.mark.parametrize("B,QH,KH,N,ctas", [OWN[2], OWN[3], OWN[5], OWN[10]])
def test_own_ctas_lengths_and_plans_of_three_bit_words(ours, oracle, B, QH, KH, N, ctas):
    """The same in 3+3, whose values' tails lie in shared memory"""
    mode, lens = "3+3", [max(1, N * i // B - 3 * i) for i in range(B)]
    q, k, v = datagen.uneven_case(21, B, QH, KH, N)
    qd = gu.bf16_tensor(q)
    c, o = ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode, capacity=N), oracle.empty(B, KH, N, mode)
    for b, n in enumerate(lens):
        row = ours.encode(gu.bf16_tensor(k[b:b + 1, :, :n]), gu.bf16_tensor(v[b:b + 1, :, :n]), mode, capacity=N)
        orow = oracle.encode(k[b:b + 1, :, :n], v[b:b + 1, :, :n], mode, capacity=N)
        for key in ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v"):
            c[key][b].copy_(row[key][0])
            o[key][b * KH:(b + 1) * KH] = orow[key]
    assert first_entry(ours, c, qd, mode, 0.0, 1).endswith(", true>")
    length, vp, passes = torch.tensor(lens, dtype=torch.int32, device="cuda"), ctypes.c_void_p, (iu.Items * 4)()
    got = ours.decode_at(c, qd, length, length_stride=1)
    torch.cuda.synchronize()
    o["tokens"] = max(lens)
    want = oracle.decode(q, o, lengths=np.array(lens, np.int32))
    for b in range(B):
        gu.check_close(gu.bits_of(got)[b], want[b], f"row of {lens[b]}")
    cfg, kc = gu.Config(B, QH, KH, 0, 0, 0, gu.FORMATS[mode][2], N, 0, 0, 0, 0, 1), ours._cache(c)
    for loops in (None, 3):
        scratch, out = ours.scratch(dict(c, tokens=N), QH), torch.empty_like(qd)
        scratch.fill_(0xFF)
        assert ours.lib.mlops_fbla_decode_at_items(ctypes.byref(cfg), vp(length.data_ptr()), vp(qd.data_ptr()), ctypes.byref(kc), vp(out.data_ptr()),
                                                   vp(scratch.data_ptr()), ctypes.c_size_t(scratch.numel()), 0, passes, 4) == 4, ours.error()
        iu.run_plan(ours.lib, passes, 4, torch.cuda.current_stream().cuda_stream, loops)
        torch.cuda.synchronize()
        assert torch.equal(out, got)


@pytest.mark.parametrize("lens", [[1, 2000, 129, 16], [300] * 3 + [1], [256, 257, 4000, 255, 31]])
def test_dense_ragged_rows(ours, oracle, lens):
    B, QH, KH, cap, mode = len(lens), 8, 2, 4096, "3+3"
    q, k, v = datagen.uneven_case(3, B, QH, KH, max(lens))
    c, o = ours.empty(B, KH, cap, mode), oracle.empty(B, KH, cap, mode)
    for b, n in enumerate(lens):
        row = ours.encode(gu.bf16_tensor(k[b:b + 1, :, :n]), gu.bf16_tensor(v[b:b + 1, :, :n]), mode, capacity=cap)
        orow = oracle.encode(k[b:b + 1, :, :n], v[b:b + 1, :, :n], mode, capacity=cap)
        for key in ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v"):
            c[key][b].copy_(row[key][0])
            o[key][b * KH:(b + 1) * KH] = orow[key]
    got = ours.decode_at(c, gu.bf16_tensor(q), torch.tensor(lens, dtype=torch.int32, device="cuda"), length_stride=1)
    torch.cuda.synchronize()
    o["tokens"] = max(lens)
    want = oracle.decode(q, o, lengths=np.array(lens, np.int32))
    for b in range(B):
        gu.check_close(gu.bits_of(got)[b], want[b], f"row {b} of {lens}")


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("QH,KH,lens,tau,scale", [(40, 40, [1, 2000, 129, 16], 0.0, 0.0), (80, 40, [1, 2000, 129, 16], 0.0, 0.0), (160, 40, [1, 2000, 129, 16], 0.0, 0.0),
                                                  (160, 40, [300] * 3 + [1], 0.0, 0.0), (120, 10, [256, 257, 1300, 255, 31], 0.0, 0.0),  # (three virtual heads per KV head)
                                                  # some sub-blocks selected; even masses: all of the short rows', none of the longest one's
                                                  (40, 40, [256, 257, 4000, 255], 5e-3, 0.0), (80, 40, [256, 257, 4000, 255], 5e-3, 0.0), (160, 40, [256, 257, 4000, 255], 5e-3, 0.0),
                                                  (40, 40, [385, 4000, 512, 31], 5e-3, 1e-3), (80, 40, [385, 4000, 512, 31], 5e-3, 1e-3), (160, 40, [385, 4000, 512, 31], 5e-3, 1e-3)])
def test_ragged_rows_dealt_over_all_ctas(ours, oracle, mode, QH, KH, lens, tau, scale):
    """Two sweeps whose groups are dealt over all CTAs (more virtual heads than SMs): rows without a closed group and of one token, in both
    formats with one, two and four queries; the plan's passes bit for bit the stream call, one CTA per item or as loops of three."""
    B, cap, vp, passes = len(lens), 4096, ctypes.c_void_p, (iu.Items * 4)()
    q, k, v = datagen.uneven_case(31 + QH, B, QH, KH, max(lens))
    c, o, qd = ours.empty(B, KH, cap, mode), oracle.empty(B, KH, cap, mode), gu.bf16_tensor(q)
    for b, n in enumerate(lens):
        row = ours.encode(gu.bf16_tensor(k[b:b + 1, :, :n]), gu.bf16_tensor(v[b:b + 1, :, :n]), mode, capacity=cap)
        for key in ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v"):
            c[key][b].copy_(row[key][0])
        orow = gu.cache_to_numpy(row)  # (the encode's bytes have tests of their own)
        for key in ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v"):
            o[key][b * KH:(b + 1) * KH] = orow[key].reshape(o[key][b * KH:(b + 1) * KH].shape)
    entry = first_entry(ours, c, qd, mode, tau, 1)
    assert entry.startswith("fbla::dense::score_item") and not entry.endswith(", true>")
    length = torch.tensor(lens, dtype=torch.int32, device="cuda")
    got = ours.decode_at(c, qd, length, length_stride=1, tau=tau, scale=scale)
    torch.cuda.synchronize()
    o["tokens"] = max(lens)
    want = oracle.decode(q, o, lengths=np.array(lens, np.int32), tau=tau, scale=scale)
    for b in range(B):
        gu.check_close(gu.bits_of(got)[b], want[b], f"row {b} of {lens}")
    cfg, kc = gu.Config(B, QH, KH, 0, scale, tau, gu.FORMATS[mode][2], cap, 0, 0, 0, 0, 1), ours._cache(c)
    scratch, out = ours.scratch(dict(c, tokens=cap), QH), torch.empty_like(qd)
    assert ours.lib.mlops_fbla_decode_at_items(ctypes.byref(cfg), vp(length.data_ptr()), vp(qd.data_ptr()), ctypes.byref(kc), vp(out.data_ptr()),
                                               vp(scratch.data_ptr()), ctypes.c_size_t(scratch.numel()), 0, passes, 4) == 4, ours.error()
    iu.run_plan(ours.lib, passes, 4, torch.cuda.current_stream().cuda_stream, 3 if scale else None)
    assert torch.equal(out, got)


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("QH,KH,cap,N,tau", [(24, 24, 14900, 385, 1e-4), (16, 8, 40000, 9001, 1e-4), (4, 1, 40000, 20011, 1e-4), (24, 2, 40000, 700, 1e-4), (32, 8, 30000, 30000, 1e-3)])
def test_a_room_beyond_one_kernel(ours, oracle, mode, QH, KH, cap, N, tau):
    """Two sweeps over few heads, dealt over all CTAs because the room is too large for a head's own: host and device lengths the same bits"""
    q, k, v = datagen.baseline_case(17 + N, 1, QH, KH, N)
    qd = gu.bf16_tensor(q)
    c = ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode, capacity=cap)
    entry = first_entry(ours, c, qd, mode, tau)
    assert entry.startswith("fbla::dense::score_item") and not entry.endswith(", true>")
    got = ours.decode(c, qd, tau=tau)
    assert torch.equal(got, ours.decode_at(c, qd, torch.tensor([N], dtype=torch.int32, device="cuda"), tau=tau))
    torch.cuda.synchronize()
    gu.check_close(gu.bits_of(got), oracle.decode(q, oracle.encode(k, v, mode, capacity=cap), tau=tau), f"{mode} {N} of {cap}")


def first_entry(ours, c, qd, mode, tau, length_stride=0):
    """the first pass of a decode's plan"""
    length, vp, passes = torch.tensor([c["tokens"]] * c["batch"], dtype=torch.int32, device="cuda"), ctypes.c_void_p, (iu.Items * 4)()
    cfg, kc = gu.Config(c["batch"], qd.shape[1], c["kv_heads"], 0, 0, tau, gu.FORMATS[mode][2], c["capacity"], 0, 0, 0, 0, length_stride), ours._cache(c)
    scratch, out = ours.scratch(dict(c, tokens=c["capacity"]), qd.shape[1]), torch.empty_like(qd)
    assert ours.lib.mlops_fbla_decode_at_items(ctypes.byref(cfg), vp(length.data_ptr()), vp(qd.data_ptr()), ctypes.byref(kc), vp(out.data_ptr()),
                                               vp(scratch.data_ptr()), ctypes.c_size_t(scratch.numel()), 0, passes, 4) == 4, ours.error()
    return passes[0].entry.decode()


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("outliers", [False, True])
@pytest.mark.parametrize("QH,N,cap,tau,first", [(8, 3000, 3000, 0.0, "dense::score_item"), (8, 3000, 400000, 0.0, "coarse_item"),  # most sub-blocks selected
                                                (8, 6000, 6000, 4e-3, "dense::score_item"), (8, 6000, 6000, 3e-2, "coarse_item"),   # few
                                                (2, 6000, 6000, 2e-3, "dense::score_item"), (2, 6000, 6000, 3e-2, "coarse_item"), (4, 20000, 20000, 3e-2, "coarse_item")])
def test_both_sides_of_the_line(ours, oracle, mode, outliers, QH, N, cap, tau, first):
    """The same rows in two sweeps and in one (a large slot, a caller's threshold), with most sub-blocks selected and with few, for values
    that spread the mass evenly and for values that do not; which way a call takes is read off its plan."""
    KH = 2
    q, k, v = datagen.baseline_case(90 + N, 1, QH, KH, N, outliers=outliers)
    qd = gu.bf16_tensor(q)
    c = ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode, capacity=cap)
    got = ours.decode(c, qd, tau=tau)
    length = torch.tensor([N], dtype=torch.int32, device="cuda")
    assert torch.equal(got, ours.decode_at(c, qd, length, tau=tau))
    torch.cuda.synchronize()
    gu.check_close(gu.bits_of(got), oracle.decode(q, oracle.encode(k, v, mode, capacity=cap), tau=tau), f"{mode} {N} of {cap}, tau {tau}")
    assert first_entry(ours, c, qd, mode, tau).startswith("fbla::" + first)


@pytest.mark.parametrize("mode", ["3+3", "4+2"])
@pytest.mark.parametrize("QH,KH,N,deal,deep", [(8, 8, 20000, 1, 0), (16, 8, 52000, 2, 0), (8, 8, 9000, 1, 1), (16, 8, 30000, 1, 1), (32, 8, 17000, 2, 1), (32, 8, 24000, 1, 1), (16, 2, 200000, 2, 0)])
def test_shapes_of_the_coarse_sweep(ours, oracle, mode, QH, KH, N, deal, deep):
    """One sweep with one, two and four queries per virtual head, twelve warps and eight, with the windows on a warp of their own and dealt by cost."""
    q, k, v = datagen.uneven_case(70 + QH, 1, QH, KH, N)
    qd, tau = gu.bf16_tensor(q), 1e-2
    c = ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode)
    assert first_entry(ours, c, qd, mode, tau).endswith(f"{deal}, {deep}>")
    got = ours.decode(c, qd, tau=tau)
    assert torch.equal(got, ours.decode_at(c, qd, torch.tensor([N], dtype=torch.int32, device="cuda"), tau=tau))
    torch.cuda.synchronize()
    gu.check_close(gu.bits_of(got), oracle.decode(q, oracle.encode(k, v, mode), tau=tau), f"{mode} {N}")


@pytest.mark.parametrize("extra", [0, 1])
def test_corrections_with_and_without_room_to_fold(ours, oracle, extra):
    """One sweep with the most (head, slice) entries whose prefix leaves the refine pass room for its row sets, and with more: a few rows of the batch"""
    mode, KH, N = "4+2", 16, 270
    limit = ours.lib.fbla_k_refine_entry_limit
    limit.restype = ctypes.c_longlong
    B = limit(4, 1) // KH + extra
    assert B > 1024 and (B * KH > limit(4, 1)) == bool(extra) and B * KH <= limit(4, 0)
    q, k, v = datagen.uneven_case(8, 3, KH, KH, N)
    rows = torch.arange(B, device="cuda") % 3
    c = ours.encode(*(gu.bf16_tensor(x)[rows].contiguous() for x in (k, v)), mode)
    qd = gu.bf16_tensor(q)[rows].contiguous()
    assert first_entry(ours, c, qd, mode, 0.0).startswith("fbla::coarse_item")
    got = ours.decode(c, qd)
    torch.cuda.synchronize()
    want = oracle.decode(q, oracle.encode(k, v, mode))
    for b in (0, 1, B // 2, B - 1):
        gu.check_close(gu.bits_of(got)[b], want[b % 3], f"row {b} of {B}")


def test_rows_of_their_own_lengths_fill_part_of_the_room(ours, oracle):
    """A room beyond the line: rows of one length are decoded in one sweep, rows of lengths of their own in two, in the scratch that the size
    query gives for either."""
    mode, QH, KH, cap, lens = "4+2", 2, 2, 22000, [300, 9000, 21000]
    q, k, v = datagen.uneven_case(12, len(lens), QH, KH, max(lens))
    qd, B = gu.bf16_tensor(q), len(lens)
    c = ours.encode(gu.bf16_tensor(k), gu.bf16_tensor(v), mode, capacity=cap)
    assert first_entry(ours, c, qd, mode, 0.0).startswith("fbla::coarse_item") and first_entry(ours, c, qd, mode, 0.0, 1).startswith("fbla::dense::score_item")
    out = ours.decode_at(c, qd, torch.tensor([max(lens)], dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    gu.check_close(gu.bits_of(out), oracle.decode(q, oracle.encode(k, v, mode, capacity=cap)), "one length")
    for b, n in enumerate(lens):  # the rows' own caches
        row = ours.encode(gu.bf16_tensor(k[b:b + 1, :, :n]), gu.bf16_tensor(v[b:b + 1, :, :n]), mode, capacity=cap)
        for key in ("coarse", "fine", "meta", "sink_k", "sink_v", "open_k", "open_v"):
            c[key][b].copy_(row[key][0])
    out = ours.decode_at(c, qd, torch.tensor(lens, dtype=torch.int32, device="cuda"), length_stride=1)
    torch.cuda.synchronize()
    for b, n in enumerate(lens):
        want = oracle.decode(q[b:b + 1], oracle.encode(k[b:b + 1, :, :n], v[b:b + 1, :, :n], mode, capacity=cap))
        gu.check_close(gu.bits_of(out)[b:b + 1], want, f"row of {n}")
