"""Host-side rules of the decode that need no GPU: how the coarse pass's work is dealt (fbla_k_decode_split), checked
through the built library, and the bench's accounting of algorithmic bytes."""
import ctypes
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LENGTHS, FIXED, COST = 0, 1, 2  # FBLA_K_DEAL_*


@pytest.fixture(scope="module")
def lib():
    if ROOT not in sys.path:
        sys.path.insert(0, ROOT)
    import __graft_entry__
    path = os.path.join(ROOT, "mlops_b200", "lib", "libmlops_attention.so")
    if not os.path.exists(path):
        __graft_entry__.build()
    return ctypes.CDLL(path)


def split_of(lib, cb, batch, kv_heads, vg, tokens):
    deal, fold = ctypes.c_int(-1), ctypes.c_int(-1)
    lib.fbla_k_decode_split_of(cb, batch, kv_heads, vg, ctypes.c_longlong(tokens), ctypes.byref(deal), ctypes.byref(fold))
    return deal.value, fold.value


@pytest.mark.parametrize("cb", [3, 4])
def test_the_deal_follows_the_groups_a_warp_would_stream(lib, cb):
    """Short rows: by the lengths. Beyond: seven + one or by cost, whichever leaves a streaming warp fewer whole groups
    (counted for 148 CTAs of eight warps), with 5 % against the deal by cost."""
    for tokens in list(range(1, 4000, 97)):
        assert split_of(lib, cb, 1, 8, 1, tokens)[0] == LENGTHS
    assert split_of(lib, cb, 256, 8, 1, 512)[0] == LENGTHS and split_of(lib, cb, 1, 8, 2, 4096)[0] == LENGTHS
    for tokens in list(range(6000, 70000, 128)) + [131072, 262144, 1 << 20, 1 << 26]:
        for batch in (1, 8, 64):
            deal, _ = split_of(lib, cb, batch, 8, 1, tokens)
            heads, S = batch * 8, (tokens + 127) // 128 - 2
            fixed = -(-heads * S // (148 * 7))
            cost = -(-(8 * heads * S + 4 * heads * 16) // (8 * 148 * 8))
            assert deal == (COST if 21 * cost < 20 * fixed else FIXED), (tokens, batch, fixed, cost)
    assert split_of(lib, cb, 1, 8, 1, 131072)[0] == COST    # 7 groups per warp instead of 8
    assert split_of(lib, cb, 8, 8, 1, 16384)[0] == FIXED    # 8 either way
    assert split_of(lib, cb, 64, 8, 1, 65280)[0] == COST


def test_rows_are_folded_per_cta_for_few_heads_only(lib):
    assert split_of(lib, 3, 1, 8, 1, 131072)[1] == 1      # 8 virtual heads, long rows
    assert split_of(lib, 4, 8, 8, 1, 16384)[1] == 0       # 64 virtual heads
    assert split_of(lib, 3, 1, 8, 1, 2048)[1] == 0        # split by the lengths: never folded
    assert split_of(lib, 4, 4, 8, 1, 65536)[1] == 1       # 32 virtual heads: the last folded size
    assert split_of(lib, 4, 4, 8, 2, 65536)[1] == 0


@pytest.mark.parametrize("qg", [1, 2, 4])
def test_two_sweeps_up_to_a_line(lib, qg):
    """Rows up to a number of tokens are decoded in two sweeps, longer ones in one; the line follows N tau, and few groups move it out."""
    two = lambda vheads, tokens, tau, batch=1: lib.fbla_k_two_sweeps(batch, vheads, qg, ctypes.c_longlong(tokens), ctypes.c_float(tau))  # noqa: E731
    for tau in (3e-4, 1e-3, 0.2):
        for vheads in (1, 2, 8, 64, 512):
            picks = [two(vheads, n, tau) for n in range(1, 300000, 997)]
            assert picks == sorted(picks, reverse=True)  # (one line: two sweeps below it)
            line = {1: 15, 2: 22, 4: 28}[qg] / tau
            assert two(vheads, int(0.99 * line), tau) and not two(vheads, int(1.6 * line), tau)
    assert two(8, 100, 3e-4, batch=1024) and not two(8, 100, 3e-4, batch=1025)  # (prefix sums of the batch in shared memory)
    assert not two(1 << 15, 1 << 20, 1e-9)                                     # (pairs of all heads below 2^29)
    assert two(8, 4096, 3e-4) and two(512, 8192, 1e-3) and not two(8, 131072, 3e-4) and not two(8, 1 << 20, 1e-3)


def test_short_rows_have_ctas_of_their_own_heads(lib):
    """As many CTAs per head as let all clusters run at once, up to a number of groups each; longer rows are dealt over all CTAs."""
    ctas = lambda vheads, tokens: lib.fbla_k_head_ctas(vheads, ctypes.c_longlong(tokens))  # noqa: E731
    for vheads in list(range(1, 160)) + [1000]:
        c = ctas(vheads, 1)
        assert (c > 0) == (vheads <= 148) and c * vheads <= 148 and c <= 16
        picks = [ctas(vheads, n) for n in range(1, 60000, 127)]
        assert set(picks) <= {c, 0} and picks == sorted(picks, reverse=True)  # (one line)
        if c:
            line = 128 * c * (16 if c == 16 else 20)
            assert ctas(vheads, line) == c and ctas(vheads, line + 1) == 0
    assert [ctas(v, 1) for v in (1, 8, 15, 16, 26, 32, 45, 64, 148)] == [16, 10, 8, 6, 5, 4, 3, 2, 1]


def head_choice(lib, vheads, qg, own_lengths, tokens, held=lambda ctas: 1000):
    fn = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_int)(lambda a, ctas: held(ctas))
    return lib.fbla_k_head_choice(None, vheads, qg, own_lengths, ctypes.c_longlong(tokens), fn)


def test_one_kernel_needs_a_device_that_holds_its_clusters(lib):
    """A device that holds fewer clusters than there are heads runs the three kernels."""
    asked = []
    for vheads in list(range(1, 150)) + [1000]:
        for tokens in (1, 4096, 30000):
            c = lib.fbla_k_head_ctas(vheads, ctypes.c_longlong(tokens))
            del asked[:]
            for held, want in [(1000, c), (vheads, c), (vheads - 1, 0), (0, 0)]:
                assert head_choice(lib, vheads, 4, 0, tokens, lambda ctas: asked.append(ctas) or held) == want
            assert asked == [c] * 4 if c else not asked  # (no query for what takes three kernels anyway)
    assert head_choice(lib, 8, 4, 0, 4096, lambda ctas: 8 if ctas <= 8 else 0) == 0  # (ten CTAs: beyond the portable size)


@pytest.mark.parametrize("qg", [1, 2, 4])
def test_rows_of_their_own_lengths_leave_one_kernel_earlier(lib, qg):
    """One line per head count, never beyond that of rows of one length; shapes on which the one kernel was measured the slower way take three."""
    line = {}
    for vheads in range(1, 149):
        for own in (0, 1):
            picks = [head_choice(lib, vheads, qg, own, n) for n in range(1, 60000, 127)]
            assert set(picks) <= {picks[0], 0} and picks[0] and picks == sorted(picks, reverse=True)
            line[vheads, own] = sum(p > 0 for p in picks)
        assert line[vheads, 1] <= line[vheads, 0] and (qg == 1 or line[vheads, 0] == sum(lib.fbla_k_head_ctas(vheads, ctypes.c_longlong(n)) > 0 for n in range(1, 60000, 127)))
    # (heads, groups per CTA) that were slower, and that were not
    slower = {4: [(75, 20), (8, 17)], 2: [(75, 17), (8, 17), (46, 17)], 1: [(8, 15), (75, 11), (80, 20), (27, 13), (46, 11), (74, 13)]}[qg]
    faster = {4: [(8, 13), (27, 20), (148, 20)], 2: [(8, 12), (33, 16), (148, 20)], 1: [(8, 9), (27, 12), (15, 14), (148, 15)]}[qg]
    for cases, chosen in ((slower, False), (faster, True)):
        for vheads, groups in cases:
            ctas = lib.fbla_k_head_ctas(vheads, ctypes.c_longlong(1))
            assert bool(head_choice(lib, vheads, qg, 1, 128 * groups * ctas)) == chosen, (vheads, groups)


def test_the_shape_follows_the_groups_a_warp_streams(lib):
    """Eight warps with a whole group in flight where twelve would not leave a warp less than three quarters of the groups."""
    deep = lambda batch, heads, qg, tokens: lib.fbla_k_decode_deep_of(batch, heads, 1, qg, ctypes.c_longlong(tokens))  # noqa: E731
    for heads, tokens, qg, want in [(8, 60000, 4, 1), (8, 150000, 4, 1), (8, 20000, 4, 1), (8, 20000, 1, 0), (8, 131072, 4, 0), (8, 266667, 4, 0),
                                    (1, 65000, 4, 1), (1, 65000, 1, 1), (8, 1 << 20, 4, 0), (1, 512, 1, 1)]:
        assert deep(1, heads, qg, tokens) == want, (heads, tokens, qg)
    assert not deep(64, 8, 4, 65536) and not deep(8, 8, 4, 131072)


class Deal(ctypes.Structure):
    _fields_ = [("cluster", ctypes.c_int), ("above", ctypes.c_int), ("tiles", ctypes.c_int)]


def test_one_launch_of_a_device_count_serves_every_chunk(lib):
    """The shares of a chunk's tiles follow from its own size; of the launches for a ceiling exactly one serves them, with all of the chunk's tiles."""
    def deal_of(heads, tiles, passes, device_count):
        d = (Deal * 2)()
        n = lib.fbla_k_attend_tc_deal(heads, tiles, passes, device_count, d)
        return [(x.cluster, x.above, x.tiles) for x in d[:n]]

    def shares(heads, tiles, passes):
        (cluster, above, _), = deal_of(heads, tiles, passes, 0)
        assert above == 0
        return cluster
    assert shares(2, 2, 95) == 7 and shares(8, 64, 512) == 1 and shares(1, 1, 23) == 1 and shares(1, 1, 24) == 2 and shares(8, 1, 1 << 19) == 8
    for heads in (1, 2, 8, 16, 70, 71, 512):
        for room in (8, 24, 25, 60, 96, 1000):
            for ceiling in (1, 2, 3, 7, 12, 36, 70, 71, 300):
                launches = deal_of(heads, ceiling, room, 1)
                for tiles in sorted({1, 2, 3, 5, 11, 12, 35, ceiling // 2, ceiling}):
                    if not 1 <= tiles <= ceiling:
                        continue
                    for passes in (1, 12, 24, room // 2, room):
                        if 1 <= passes <= room:
                            n = shares(heads, tiles, passes)
                            serving = [x for x in launches if x[1] < n <= x[0]]
                            assert len(serving) == 1 and serving[0][2] >= tiles, (heads, room, ceiling, tiles, passes, launches)


def test_bench_accounts_the_bytes_the_way_the_reference_bench_does():
    """Algorithmic bytes of a decode: per closed (KV head, group) 8 coarse records + 1 KiB of metadata, 512 B per BF16
    window token, 3 072 B per refined (KV head, sub-block) (attention/fbla/bench/bench_fbla.cu:136-141)."""
    if ROOT not in sys.path:
        sys.path.insert(0, ROOT)
    import bench
    assert set(bench.NCU_TRAFFIC) <= set(bench.WORKLOADS) and set(bench.SUBS) <= set(bench.WORKLOADS)
    assert bench.WORKLOADS["decode_128k"]["tokens"] == 131072 and bench.WORKLOADS["decode_128k"]["mode"] == "3+3"
    total, parts = bench.decode_bytes(dict(batch=1, kv_heads=8, tokens=131072, mode="3+3"), 0.0)
    groups = 131072 // 128 - 2
    assert parts["coarse_and_meta"] == 8 * groups * (8 * 1536 + 1024)
    assert parts["bf16_windows"] == 8 * 256 * 512 and total == parts["coarse_and_meta"] + parts["bf16_windows"]
    total, parts = bench.decode_bytes(dict(batch=8, kv_heads=8, tokens=16384, mode="4+2"), 0.5)
    assert parts["coarse_and_meta"] == 64 * 126 * (8 * 2048 + 1024) and parts["refine"] == 0.5 * 64 * 126 * 8 * 3072


def test_reference_arm_prints_the_contract_line_without_a_gpu():
    """`bench.py --impl reference` is the oracle's port of the reference's host model on the host cores: it needs no GPU,
    and its one JSON line carries the keys the measurement contract names."""
    import json
    import subprocess
    run = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0"],
                         capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert run.returncode == 0, run.stderr[-2000:]
    lines = [l for l in run.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["metric"] == "decode_tokens_per_s" and d["unit"] == "tokens/s" and d["higher_is_better"] is True
    assert d["config"]["tokens"] == 131072 and d["config"]["mode"] == "3+3" and d["value"] > 0
    assert d["cpu_baseline"]["kind"] == "port" and d["cpu_baseline"]["cores"] >= 1 and d["cpu_baseline"]["value"] == d["value"]
    assert d["e2e"] == dict(value=d["value"], unit="tokens/s", h2d_bytes_per_step=0, d2h_bytes_per_step=0)
