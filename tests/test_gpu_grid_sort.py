"""Sorts between the cluster's sizes and the general route's: one resident grid."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from thrust_b200 import datagen as dg
from gpu_util import dev, host, rand_of

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# both sides of the cluster's limit, of two and four rows per warp on 148 SMs, of a last CTA with few items, of the route's limits
SIZES = [32768, 32769, 33791, 65536, 100003, 148 * 1024, 148 * 1024 + 1, 148 * 2048 - 511, 148 * 2048 + 33, 288 << 10, (288 << 10) + 1, (448 << 10) - 31, (448 << 10) + 1]


@pytest.mark.parametrize("n", SIZES)
def test_pairs(tb, port, n):
    for kt, vt, desc in [(np.uint32, np.uint32, False), (np.int64, np.uint64, True), (np.float32, np.uint64, False), (np.uint64, np.uint32, False)]:
        k = rand_of(kt, n, 61)
        if kt is np.uint64:
            k >>= np.uint64(24)                      # places that all keys share are left out
        v = np.arange(n, dtype=vt)
        dk, dv = dev(k), dev(v)
        tb.sort_by_key(dk, dv, descending=desc)
        wk, wv = port.sort_by_key(k, v, desc)
        assert np.array_equal(host(dk), wk) and np.array_equal(host(dv), wv), (kt, vt)


@pytest.mark.parametrize("n", SIZES[::3])
def test_keys(tb, port, n):
    for dt in (np.int8, np.uint16, np.int32, np.float64):
        for k in (rand_of(dt, n, 62), rand_of(dt, n, 63, small=True), np.full(n, 3, dtype=dt), np.sort(rand_of(dt, n, 64))[::-1].copy()):
            for desc in (False, True):
                d = dev(k)
                tb.sort(d, descending=desc)
                wk, _ = port.sort_by_key(k, None, desc)
                assert np.array_equal(host(d), wk), (dt, desc)


def test_some_bits_only(tb):
    n = 77777
    k, v = (dg.rand64(65, n) >> np.uint64(32)).astype(np.uint32), np.arange(n, dtype=np.uint32)
    for b0, b1 in [(8, 16), (0, 24), (16, 32)]:
        dk, dv = dev(k), dev(v)
        tb.sort_by_key(dk, dv, begin_bit=b0, end_bit=b1)
        order = np.argsort((k >> np.uint32(b0)) & np.uint32((1 << (b1 - b0)) - 1), kind="stable")
        assert np.array_equal(host(dk), k[order]) and np.array_equal(host(dv), v[order]), (b0, b1)


def test_a_meeting_that_runs_out(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.isfile(nvcc):
        pytest.skip("nvcc is not available on this machine")
    exe = str(tmp_path / "grid_sort_wait_test")
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O2", "-DTB200_TEST_HOOKS", "-DTB200_SPIN_LIMIT=65536",
                        "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "grid_sort_wait_test.cu"), "-o", exe],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "all checks passed" in r.stdout, r.stdout + r.stderr
