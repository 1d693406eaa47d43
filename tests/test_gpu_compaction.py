"""Parity of copy_if, partition, unique and reduce_by_key (through the C ABI) with the CPU oracle."""
import numpy as np
import pytest
import torch

from thrust_b200 import datagen as dg
from gpu_util import ALL, EDGE_SIZES, WIDE, dev, host, misaligned, rand_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", EDGE_SIZES)
def test_copy_if_and_partition_bit_exact(tb, oracles, n):
    x = dg.compaction_input(n)
    got = host(tb.copy_if(dev(x), "mod_eq", 2, 0))
    gt, gf = tb.partition_copy(dev(x), "mod_eq", 2, 0)
    d = dev(x)
    split = tb.partition(d, "mod_eq", 2, 0)
    for o in oracles:
        assert np.array_equal(got, o.copy_if(x, "mod_eq", 2, 0))
        ot, of = o.partition_copy(x, "mod_eq", 2, 0)
        assert np.array_equal(host(gt), ot) and np.array_equal(host(gf), of)
        sd, sc = o.stable_partition(x, "mod_eq", 2, 0)
        assert split == sc and np.array_equal(host(d), sd)
        # thrust::partition contract: split point and selected half exact, rejected half as a multiset
        # (testing/partition.cu:309-312 sorts both halves before comparing)
        ud, uc = o.partition(x, "mod_eq", 2, 0)
        assert split == uc and np.array_equal(host(d)[:split], ud[:uc])
        assert np.array_equal(np.sort(host(d)[split:]), np.sort(ud[uc:]))


def test_copy_if_types_predicates_stencils(tb, port):
    n = 33333
    for dt in ALL:
        x = rand_of(dt, n, 61, small=True)
        preds = [("ne", 3, 0), ("lt", 3, 0), ("ge", 2, 0)] + ([("mod_eq", 3, 1)] if np.dtype(dt).kind != "f" else [])
        for pred, a, b in preds:
            assert np.array_equal(host(tb.copy_if(dev(x), pred, a, b)), port.copy_if(x, pred, a, b)), (dt, pred)
            gt, gf = tb.partition_copy(dev(x), pred, a, b)
            ot, of = port.partition_copy(x, pred, a, b)
            assert np.array_equal(host(gt), ot) and np.array_equal(host(gf), of), (dt, pred)
            d = dev(x)
            split = tb.stable_partition(d, pred, a, b)
            sd, sc = port.stable_partition(x, pred, a, b)
            assert split == sc and np.array_equal(host(d), sd), (dt, pred)
        for st_dt in (np.uint8, np.int32):
            st = rand_of(st_dt, n, 62, small=True)
            assert np.array_equal(host(tb.copy_if(dev(x), "ne", 0, 0, stencil=dev(st))), port.copy_if(x, "ne", 0, 0, stencil=st)), (dt, st_dt)
            gt, gf = tb.partition_copy(dev(x), "ge", 3, 0, stencil=dev(st))
            keep = st >= 3
            assert np.array_equal(host(gt), x[keep]) and np.array_equal(host(gf), x[~keep]), (dt, st_dt)


def test_copy_if_extremes_in_place_misaligned(tb, port):
    x = dg.compaction_input(100001)
    assert tb.copy_if(dev(x), "lt", 0, 0).numel() == 0                        # nothing selected
    assert np.array_equal(host(tb.copy_if(dev(x), "ge", 0, 0)), x)            # everything selected
    d = dev(x)
    out = tb.copy_if(d, "mod_eq", 2, 0, out=d)                                # result == first (remove_if, remove.h:38-65)
    assert np.array_equal(host(out), port.copy_if(x, "mod_eq", 2, 0))
    assert np.array_equal(host(tb.copy_if(misaligned(x, 3), "mod_eq", 2, 0)), port.copy_if(x, "mod_eq", 2, 0))


@pytest.mark.parametrize("dt", [np.int32, np.int64])
def test_compaction_large_bit_exact(tb, oracles, dt):
    """2^25 + 12345 items (thousands of tiles, a partial last one), out of place and in place."""
    n = (1 << 25) + 12345
    x = dg.compaction_input(n).astype(dt)
    keys = dg.run_keys(n).astype(dt)
    stencil = (dg.scan_input_i32(n, 9) & 3).astype(np.int32)
    got = host(tb.copy_if(dev(x), "mod_eq", 3, 1))
    got_st = host(tb.copy_if(dev(x), "ne", 0, 0, stencil=dev(stencil)))
    gt, gf = tb.partition_copy(dev(x), "lt", 1 << 20, 0)
    d = dev(x)
    split = tb.partition(d, "mod_eq", 2, 0)
    u = host(tb.unique_copy(dev(keys)))
    dk = dev(keys)
    ui = host(tb.unique(dk))
    for o in oracles:
        assert np.array_equal(got, o.copy_if(x, "mod_eq", 3, 1))
        assert np.array_equal(got_st, o.copy_if(x, "ne", 0, 0, stencil=stencil))
        ot, of = o.partition_copy(x, "lt", 1 << 20, 0)
        assert np.array_equal(host(gt), ot) and np.array_equal(host(gf), of)
        sd, sc = o.stable_partition(x, "mod_eq", 2, 0)
        assert split == sc and np.array_equal(host(d), sd)
        ref_u = o.unique_copy(keys)
        assert np.array_equal(u, ref_u) and np.array_equal(ui, ref_u)


@pytest.mark.parametrize("kt,vt", [(np.int32, np.int32), (np.uint32, np.float32), (np.int64, np.int64), (np.uint64, np.float64), (np.int32, np.int64)])
def test_reduce_by_key_large_bit_exact(tb, oracles, kt, vt):
    """2^25 + 12345 items: keys and values of one size take the two-pass streaming kernels, mixed
    sizes the single-pass one; the last row of the input is partial.  Integer sums, minima and the
    first-of-run selection of unique_by_key are exact; floating-point values are small integers here,
    so their sums are exact too."""
    n = (1 << 25) + 12345
    keys = dg.run_keys(n).astype(kt)
    vals = (dg.scan_input_i32(n, 7) % 1000).astype(vt)
    ko, vo = tb.reduce_by_key(dev(keys), dev(vals))
    km, vm = tb.reduce_by_key(dev(keys), dev(vals), op="min")
    uk, uv = (None, None)
    if np.dtype(vt).itemsize in (4, 8):
        uk, uv = tb.unique_by_key_copy(dev(keys), dev(vals))
    dk, dv = dev(keys), dev(vals)
    ik, iv = tb.unique_by_key(dk, dv)                                          # in place: single-pass kernel
    for o in oracles:
        rk, rv = o.reduce_by_key(keys, vals)
        assert np.array_equal(host(ko), rk) and np.array_equal(host(vo), rv)
        mk, mv = o.reduce_by_key(keys, vals, "min")
        assert np.array_equal(host(km), mk) and np.array_equal(host(vm), mv)
        fk, fv = o.unique_by_key_copy(keys, vals)
        assert np.array_equal(host(uk), fk) and np.array_equal(host(uv), fv)
        assert np.array_equal(host(ik), fk) and np.array_equal(host(iv), fv)


@pytest.mark.parametrize("n", EDGE_SIZES)
def test_unique_and_reduce_by_key(tb, oracles, n):
    keys = dg.run_keys(n)
    ivals = dg.scan_input_i32(n, 7)
    fvals = dg.run_values_f32(n)
    u = host(tb.unique_copy(dev(keys)))
    d = dev(keys)
    ui = host(tb.unique(d))                                                   # in place, unique.h:772
    ko, vo = tb.reduce_by_key(dev(keys), dev(ivals))
    kf, vf = tb.reduce_by_key(dev(keys), dev(fvals))
    for o in oracles:
        ref_u = o.unique_copy(keys)
        assert np.array_equal(u, ref_u) and np.array_equal(ui, ref_u)
        rk, rv = o.reduce_by_key(keys, ivals)
        assert np.array_equal(host(ko), rk) and np.array_equal(host(vo), rv)
        # fp32 values: keys and run count exact, sums within 1e-6 relative of the fp64 yardstick
        yk, yv = o.reduce_by_key_f32_via_f64(keys, fvals)
        assert np.array_equal(host(kf), yk)
        assert np.allclose(host(vf), yv, rtol=1e-6, atol=0)


def test_unique_rbk_types_and_shapes(tb, port):
    n = 40009
    for dt in ALL:
        x = rand_of(dt, n, 63, small=True)
        assert np.array_equal(host(tb.unique_copy(dev(x))), port.unique_copy(x)), dt
        for vt in WIDE:
            vals = rand_of(vt, n, 64, small=True)
            for op in ("plus", "min", "max"):
                gk, gv = tb.reduce_by_key(dev(x), dev(vals), op)
                rk, rv = port.reduce_by_key(x, vals, op)
                assert np.array_equal(host(gk), rk) and np.array_equal(host(gv), rv), (dt, vt, op)
    # one long run spanning many tiles, all-distinct keys, alternating keys
    for keys in (np.zeros(50000, np.int32), np.arange(50000, dtype=np.int32), (np.arange(50000) % 2).astype(np.int32)):
        vals = np.ones(keys.size, np.int64)
        gk, gv = tb.reduce_by_key(dev(keys), dev(vals))
        rk, rv = port.reduce_by_key(keys, vals)
        assert np.array_equal(host(gk), rk) and np.array_equal(host(gv), rv)
        assert np.array_equal(host(tb.unique_copy(dev(keys))), port.unique_copy(keys))
    f = np.array([0.0, -0.0, 1.0, np.nan, np.nan, 2.0, 2.0], np.float32)     # IEEE equality: -0 == 0, NaN != NaN
    assert host(tb.unique_copy(dev(f))).size == port.unique_copy(f).size == 5


def test_golden_compaction(tb, golden):
    for n in (1, 777, 12345):
        c = golden[f"compact_in_{n}"]
        assert np.array_equal(host(tb.copy_if(dev(c), "mod_eq", 2, 0)), golden[f"copy_if_out_{n}"])
        d = dev(c)
        assert tb.stable_partition(d, "mod_eq", 2, 0) == golden[f"partition_count_{n}"]
        assert np.array_equal(host(d), golden[f"stable_partition_out_{n}"])
        assert np.array_equal(host(tb.unique_copy(dev(golden[f"run_keys_{n}"]))), golden[f"unique_out_{n}"])
        gk, gv = tb.reduce_by_key(dev(golden[f"run_keys_{n}"]), dev(golden[f"run_vals_{n}"]))
        assert np.array_equal(host(gk), golden[f"rbk_keys_out_{n}"]) and np.array_equal(host(gv), golden[f"rbk_vals_out_{n}"])


def test_full_size_compaction_properties(tb):
    """2^28 elements: copy_if output equals a boolean-mask selection; partition halves concatenate to
    a stable split; unique of run keys is 0..runs-1; reduce_by_key of ones gives the run lengths."""
    n = 1 << 28
    x = dev(dg.compaction_input(n))
    sel = tb.copy_if(x, "mod_eq", 2, 0)
    mask = (x & 1) == 0
    assert sel.numel() == int(mask.sum()) and torch.equal(sel, x[mask])
    del sel
    d = x.clone()
    split = tb.partition(d, "mod_eq", 2, 0)
    assert split == int(mask.sum()) and torch.equal(d[:split], x[mask]) and torch.equal(d[split:], x[~mask])
    del d, x, mask
    keys = dev(dg.run_keys(n))
    runs = int(keys[-1]) + 1
    u = tb.unique_copy(keys)
    assert u.numel() == runs and torch.equal(u, torch.arange(runs, dtype=torch.int32, device="cuda"))
    del u
    ones = torch.ones(n, dtype=torch.int32, device="cuda")
    gk, gv = tb.reduce_by_key(keys, ones)
    assert gk.numel() == runs and int(gv.sum()) == n
    assert torch.equal(gv, torch.bincount(keys, minlength=runs).to(torch.int32))


def test_full_size_reduce_by_key_fp32(tb):
    """reduce_by_key at the benchmark size with its fp32 values in [0, 1): output keys and run count
    exact (against bincount), every segment sum within 1e-6 relative of an fp64 segment sum."""
    n = 1 << 28
    keys = dev(dg.run_keys(n))
    vals = dev(dg.run_values_f32(n))
    runs = int(keys[-1]) + 1
    gk, gv = tb.reduce_by_key(keys, vals)
    assert gk.numel() == runs and gv.numel() == runs
    assert torch.equal(gk, torch.arange(runs, dtype=torch.int32, device="cuda"))
    del gk
    yard = torch.zeros(runs, dtype=torch.float64, device="cuda")
    step = 1 << 26                                       # bounded temporaries
    for lo in range(0, n, step):
        yard.index_add_(0, keys[lo:lo + step].long(), vals[lo:lo + step].double())
    err = (gv.double() - yard).abs() / yard.clamp(min=1e-30)
    assert float(err.max()) < 1e-6, float(err.max())


@pytest.mark.parametrize("items", [1 << 18, (1 << 20) - 1, (1 << 20) + 1, 148 * 8192, 148 * 8192 + 1, 3 * 148 * 8192 + 4099])
def test_compaction_pipeline_edges(tb, port, items):
    """Around the sizes where the pipeline starts, whole and ragged rounds of 148 tiles, nothing / few / half / all kept, and
    outputs that start off a 16-byte boundary."""
    for dt in (np.int32, np.int64, np.float32):
        n = items * 4 // np.dtype(dt).itemsize
        x = (dg.rand64(61, n) % np.uint64(1 << 20)).astype(dt)
        for bound in (0, 1 << 10, 1 << 19, 1 << 20):
            want = port.copy_if(x, "lt", bound, 0)
            out = misaligned(np.zeros(n, dt), 1)
            assert np.array_equal(host(tb.copy_if(dev(x), "lt", bound, 0, out=out)), want), (dt, bound)
            sel, rej = tb.partition_copy(dev(x), "lt", bound, 0)
            assert np.array_equal(host(sel), want) and np.array_equal(host(rej), x[x >= bound]), (dt, bound)
            d = dev(x)
            assert tb.partition(d, "lt", bound, 0) == want.size
            assert np.array_equal(host(d), np.concatenate([want, x[x >= bound]])), (dt, bound)
        for run in (1, 3, 1000, n + 1):
            r = (np.arange(n) // run).astype(dt)
            assert np.array_equal(host(tb.unique_copy(dev(r))), port.unique_copy(r)), (dt, run)


@pytest.mark.parametrize("items", [131071, 131073, 148 * 4096, 148 * 4096 + 1, 3 * 148 * 4096 + 2050])
def test_reduce_by_key_pipeline_edges(tb, port, items):
    """Around the size where the pipeline starts, whole and ragged rounds of 148 tiles, one run, runs that end with a tile
    and runs of one item; mixed sizes of keys and values.  Doubles hold whole numbers, so their sums are exact."""
    for kt, vt in [(np.int32, np.int32), (np.uint32, np.float64), (np.int64, np.int32), (np.uint64, np.float64), (np.float32, np.int64)]:
        v = dg.scan_input_i32(items, 7).astype(vt)
        for run in (1, 2, 37, 4096, items + 1):
            k = (np.arange(items) // run).astype(kt)
            for op in ("plus", "max"):
                gk, gv = tb.reduce_by_key(dev(k), dev(v), op=op)
                wk, wv = port.reduce_by_key(k, v, op)
                assert np.array_equal(host(gk), wk) and np.array_equal(host(gv), wv), (kt, vt, run, op)


@pytest.mark.parametrize("kt,vt", [(np.int32, np.float32), (np.int64, np.float64)])
def test_reduce_by_key_float_min_max_of_nans(tb, kt, vt):
    """Runs of nothing but NaNs reduce to NaN wherever they lie -- at the ends of rows, warps' parts and tiles, over
    several of them -- and never to an infinity that is not in the input; runs without NaNs are exact."""
    n = (1 << 24) + 4099
    for run in (1, 2, 7, 512, 4096, 10000):
        k = (np.arange(n) // run).astype(kt)
        v = (dg.rand64(53, n) % np.uint64(1 << 20)).astype(vt)
        nan_run = dg.rand64(54, int(k[-1]) + 1) % np.uint64(3) == 0
        v[nan_run[k]] = np.nan
        starts = np.arange(0, n, run)
        for op, fold in (("min", np.minimum), ("max", np.maximum)):
            gk, gv = tb.reduce_by_key(dev(k), dev(v), op=op)
            assert np.array_equal(host(gk), np.arange(starts.size).astype(kt)), (run, op)
            assert np.array_equal(host(gv), fold.reduceat(v, starts), equal_nan=True), (run, op)


@pytest.mark.parametrize("keep", [0.5, 0.97, 1.0])
def test_in_place_partition_over_its_own_input(tb, keep):
    """Kept items land on what other CTAs read just before; with nearly all kept, on their neighbours' tiles.  Many passes, a
    copy running beside them on another stream."""
    n = (1 << 24) + 4099
    x = dev((dg.rand64(62, n) % np.uint64(1 << 20)).astype(np.int32))
    bound = int(keep * (1 << 20))
    want = torch.cat([x[x < bound], x[x >= bound]])
    d, other, side = torch.empty_like(x), torch.empty_like(x), torch.cuda.Stream()
    for _ in range(50):
        d.copy_(x)
        with torch.cuda.stream(side):
            other.copy_(x)
        assert tb.partition(d, "lt", bound, 0) == int((x < bound).sum())
        assert torch.equal(d, want)
