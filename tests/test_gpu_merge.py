"""Parity of merge / merge_by_key (through the C ABI) with the CPU oracle."""
import numpy as np
import pytest
import torch

from thrust_b200 import datagen as dg
from gpu_util import dev, host, misaligned, rand_of

pytestmark = pytest.mark.gpu
KEY_TYPES = [np.int32, np.uint32, np.float32, np.int64, np.uint64, np.float64]


@pytest.mark.parametrize("n", [0, 1, 2, 33, 2815, 2816, 2817, 3839, 3841, 8193, 65536 + 17, (1 << 20) + 3])
def test_merge_by_key_u64_bit_exact_and_stable(tb, oracles, n):
    # testing/merge_by_key.cu:129-196 splits n unevenly, including an empty side
    for na, nb in [(n, n), (n, n // 3), (0, n), (n, 0), (n // 9, n)]:
        a = np.sort((dg.rand64(4, na) >> np.uint64(52)).astype(np.uint64))     # 12-bit keys: ties between A and B
        b = np.sort((dg.rand64(5, nb) >> np.uint64(52)).astype(np.uint64))
        va = np.arange(na, dtype=np.uint32)
        vb = np.arange(nb, dtype=np.uint32) + np.uint32(1 << 27)               # payload tells A from B
        ko, vo = tb.merge_by_key(dev(a), dev(b), dev(va), dev(vb))
        for o in oracles:
            rk, rv = o.merge_by_key(a, b, va, vb)
            assert np.array_equal(host(ko), rk) and np.array_equal(host(vo), rv), (na, nb)


def test_merge_types_orders_payloads(tb, port):
    n = 30011
    for dt in KEY_TYPES:
        for desc in (False, True):
            a, _ = port.sort_by_key(rand_of(dt, n, 71, small=True), None, desc)
            b, _ = port.sort_by_key(rand_of(dt, n // 2, 72, small=True), None, desc)
            rk, _ = port.merge_by_key(a, b, None, None, desc)
            assert np.array_equal(host(tb.merge(dev(a), dev(b), desc)), rk), (dt, desc)
            for vt in (np.uint32, np.uint64):
                va, vb = np.arange(a.size, dtype=vt), np.arange(b.size, dtype=vt) + vt(1 << 30)
                ko, vo = tb.merge_by_key(dev(a), dev(b), dev(va), dev(vb), desc)
                rk, rv = port.merge_by_key(a, b, va, vb, desc)
                assert np.array_equal(host(ko), rk) and np.array_equal(host(vo), rv), (dt, vt, desc)


def test_golden_merge(tb, golden):
    for n in (1, 777, 12345):
        a, b = golden[f"merge_a_{n}"], golden[f"merge_b_{n}"]
        va = np.arange(a.size, dtype=np.uint32)
        vb = np.arange(b.size, dtype=np.uint32) + np.uint32(1 << 27)
        ko, vo = tb.merge_by_key(dev(a), dev(b), dev(va), dev(vb))
        assert np.array_equal(host(ko), golden[f"merge_keys_out_{n}"]) and np.array_equal(host(vo), golden[f"merge_vals_out_{n}"])


def test_full_size_merge_properties(tb):
    """2 x 2^27 (u64 key, u32 payload): output sorted, each input a subsequence (payloads of A and of
    B each appear in increasing order), ties put A first."""
    n = 1 << 27
    a = dev(dg.merge_keys_u64(n, 4))
    b = dev(dg.merge_keys_u64(n, 5))
    va = torch.arange(n, dtype=torch.int32, device="cuda")
    vb = va + n
    ko, vo = tb.merge_by_key(a, b, va, vb)
    ki = ko.view(torch.int64)                                  # keys < 2^48: signed view keeps the order
    assert bool((ki[1:] >= ki[:-1]).all())
    from_a = vo < n
    assert torch.equal(vo[from_a], va) and torch.equal(vo[~from_a], vb)
    assert torch.equal(ki[from_a], a.view(torch.int64)) and torch.equal(ki[~from_a], b.view(torch.int64))
    ties = ki[1:] == ki[:-1]
    assert bool((~(from_a[1:] & ~from_a[:-1] & ties)).all())   # never B directly before an equal A


@pytest.mark.parametrize("num_runs", [1, 2, 3, 5, 8])
def test_merge_runs_tree(tb, port, num_runs):
    """tb200_merge_runs: many sorted runs in one call, equal to folding the oracle's two-way merge
    over them in order (ties keep the earlier run first)."""
    import ctypes as C
    from thrust_b200 import api
    lib = tb._lib.load()
    runs_k, runs_v, dk, dv = [], [], [], []
    for r in range(num_runs):
        n = [30011, 0, 4097, 1, 70001, 2816, 5, 12345][r]
        k = np.sort((dg.rand64(80 + r, n) >> np.uint64(54)).astype(np.uint32))       # 10-bit keys: ties across runs
        v = (np.arange(n, dtype=np.uint32) + np.uint32(r << 24))
        runs_k.append(k); runs_v.append(v); dk.append(dev(k)); dv.append(dev(v))
    total = sum(k.size for k in runs_k)
    wk, wv = runs_k[0], runs_v[0]
    for r in range(1, num_runs):
        wk, wv = port.merge_by_key(wk, runs_k[r], wv, runs_v[r])
    ko = torch.empty(total, dtype=torch.uint32, device="cuda"); kt = torch.empty_like(ko)
    vo = torch.empty(total, dtype=torch.uint32, device="cuda"); vt = torch.empty_like(vo)
    kp = (C.c_void_p * num_runs)(*[t.data_ptr() for t in dk])
    vp = (C.c_void_p * num_runs)(*[t.data_ptr() for t in dv])
    cn = (C.c_size_t * num_runs)(*[t.numel() for t in dk])
    ws = api._call_with_ws("merge", "tb200_merge_runs", kp, vp, cn, num_runs, api._ptr(ko), api._ptr(vo), api._ptr(kt), api._ptr(vt), 5, 4, 0)
    api._sync_and_check(ws, "merge_runs")
    assert np.array_equal(host(ko), wk) and np.array_equal(host(vo), wv)


@pytest.mark.parametrize("shift", [(0, 1), (1, 0), (3, 2), (1, 3)])
@pytest.mark.parametrize("n", [1, 5, 1023, 2047, 2048, 2049, 6151])
def test_merge_of_slices_at_any_alignment(tb, port, shift, n):
    """Inputs that start anywhere between two 16-byte boundaries, tiles of 2048 outputs and their remainders."""
    for dt, vt in [(np.uint32, np.uint32), (np.uint64, np.uint32), (np.uint32, np.uint64), (np.float64, np.uint64)]:
        a, _ = port.sort_by_key(rand_of(dt, n, 91, small=True), None, False)
        b, _ = port.sort_by_key(rand_of(dt, n // 2 + 1, 92), None, False)
        va, vb = np.arange(a.size, dtype=vt), np.arange(b.size, dtype=vt) + vt(1 << 30)
        args = [misaligned(x, (s * (q + 1)) % 4) for q, (x, s) in enumerate([(a, shift[0]), (b, shift[1]), (va, shift[1]), (vb, shift[0])])]
        ko, vo = tb.merge_by_key(*args)
        rk, rv = port.merge_by_key(a, b, va, vb)
        assert np.array_equal(host(ko), rk) and np.array_equal(host(vo), rv), (dt, vt)
        assert np.array_equal(host(tb.merge(args[0], args[1])), rk), dt


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_merge_of_keys_with_nans_ends(tb, port, dt):
    """Keys that are NaN have no order: the call gives some order or reports that its tiles disagree, and the next call
    on the same workspace is right."""
    n = 200003
    a, b = np.sort(rand_of(dt, n, 93)), np.sort(rand_of(dt, n // 2, 94))
    va, vb = np.arange(n, dtype=np.uint32), np.arange(n // 2, dtype=np.uint32) + np.uint32(1 << 30)
    for share in (0.002, 0.02, 0.1):
        an, bn = a.copy(), b.copy()
        an[dg.rand64(95, n) % np.uint64(1000) < int(1000 * share)] = np.nan
        bn[dg.rand64(96, n // 2) % np.uint64(1000) < int(1000 * share)] = np.nan
        for call in (lambda: tb.merge_by_key(dev(an), dev(bn), dev(va), dev(vb)), lambda: tb.stable_sort_zip_by_first(dev(an[dg.rand64(97, n) % np.uint64(n)]), dev(va))):
            try:
                assert call()[0].numel() >= n
            except tb.api.Tb200Error as e:
                assert "status 2" in str(e)
        ko, vo = tb.merge_by_key(dev(a), dev(b), dev(va), dev(vb))
        rk, rv = port.merge_by_key(a, b, va, vb)
        assert np.array_equal(host(ko), rk) and np.array_equal(host(vo), rv)


@pytest.mark.parametrize("n", [4096 * 2048 + 1, 256 * 17 * 2048, 256 * 18 * 2048 + 2047])
def test_merge_splits_of_many_tiles(tb, port, n):
    """More than 4096 tiles of 2048 outputs: a thread per tile between the splits of its group of 256.  Even and uneven mixes,
    ties, ranges that do not overlap, one side empty or a single item; whole groups and a last group of one tile."""
    rnd = lambda seed, m, bits: np.sort((dg.rand64(seed, m) >> np.uint64(64 - bits)).astype(np.uint32))  # noqa: E731
    third, high = n // 3, np.uint32(1 << 31)
    for a, b in [(rnd(1, n - third, 31), rnd(2, third, 31)), (rnd(3, n // 2, 2), rnd(4, n - n // 2, 3)), (rnd(5, third, 30) + high, rnd(6, n - third, 30)),
                 (rnd(7, n - 1, 30), rnd(8, 1, 30)), (rnd(9, 0, 30), rnd(10, n, 30)),
                 (np.sort(rnd(11, n // 2, 30) // np.uint32(1 << 20) * np.uint32(1 << 10)), rnd(12, n - n // 2, 20))]:
        va, vb = np.arange(a.size, dtype=np.uint32), np.arange(b.size, dtype=np.uint32) + high
        ko, vo = tb.merge_by_key(dev(a), dev(b), dev(va), dev(vb))
        rk, rv = port.merge_by_key(a, b, va, vb)
        assert np.array_equal(host(ko), rk) and np.array_equal(host(vo), rv), (a.size, b.size)


def test_merge_sort_splits_of_many_tiles(tb, port):
    """The same in the passes of a sort: pairs of fewer and of more tiles than a group, a short last pair."""
    n = 4200 * 2048 + 777
    for bits in (32, 3):
        k, v = (dg.rand64(13, n) >> np.uint64(64 - bits)).astype(np.uint32), np.arange(n, dtype=np.uint32)
        dk, dv = dev(k), dev(v)
        tb.merge_sort_by_key(dk, dv)
        rk, rv = port.sort_by_key(k, v)
        assert np.array_equal(host(dk), rk) and np.array_equal(host(dv), rv)
