"""A bounded wait that runs out: the kernel returns, the status word says so, the host raises.

Every inter-CTA wait in the library gives up after a fixed number of polls, records status 1 in the
workspace header and carries on, so a broken launch can never hang the device.  This test makes one
run out without faulting or hanging anything: it loads the TEST build of the scan entry points
(thrust_b200.build.build_shortwait: 64 polls instead of 2^23) and switches on its hook that makes
the first tile of a single-pass scan withhold its descriptor.  Every index stays in bounds; the later
tiles' polls of tile 0 simply expire after a few microseconds.  Afterwards the same workspace serves
an ordinary call again."""
import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_lookback_timeout_is_reported_and_recoverable(tb, port, monkeypatch):
    import torch
    from thrust_b200 import _lib, api, build, datagen as dg
    if not os.path.isfile(build.SHORTWAIT_LIB):
        pytest.fail("%s is missing -- python -m thrust_b200.build makes it" % build.SHORTWAIT_LIB)
    short = _lib.load_partial(build.SHORTWAIT_LIB)
    short.tb200_test_hooks.argtypes = [C.c_uint]
    short.tb200_test_hooks.restype = C.c_int
    n = 5 * 8192 + 123                                   # six tiles of the single-pass kernel
    x_h = dg.scan_input_i32(n)
    x = torch.from_numpy(x_h).cuda()
    out = torch.empty_like(x)
    need = C.c_size_t(0)
    assert short.tb200_inclusive_scan(None, None, n, 4, 0, None, None, C.byref(need), None) == 0
    ws = torch.zeros(need.value, dtype=torch.uint8, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    status = C.c_uint(7)

    # 1. the wait runs out: the call itself succeeds (it only enqueues), the kernel returns, status = 1
    assert short.tb200_test_hooks(1) == 0
    assert short.tb200_inclusive_scan(p(x), p(out), n, 4, 0, None, p(ws), C.byref(need), None) == 0
    assert short.tb200_workspace_status(p(ws), None, C.byref(status)) == 0
    assert status.value == 1
    torch.cuda.synchronize()                              # the context is alive and well

    # 2. the host side of the library turns that status into an exception
    monkeypatch.setattr(_lib, "_lib", short)
    with pytest.raises(api.Tb200Error):
        tb.inclusive_scan(x)

    # 3. hook off: the same workspace and the same (short-wait) kernels give the right answer again
    assert short.tb200_test_hooks(0) == 0
    got = tb.inclusive_scan(x)
    assert np.array_equal(got.cpu().numpy(), port.inclusive_scan(x_h))
    assert short.tb200_inclusive_scan(p(x), p(out), n, 4, 0, None, p(ws), C.byref(need), None) == 0
    assert short.tb200_workspace_status(p(ws), None, C.byref(status)) == 0 and status.value == 0
    assert np.array_equal(out.cpu().numpy(), port.inclusive_scan(x_h))


def test_waits_of_the_pipelines_and_the_merge_run_out(tb, tmp_path):
    """tests/cpp/bounded_waits_test.cu, built here with the test hooks and short waits: a withheld tile descriptor in the
    scan, compaction, partition and reduce_by_key pipelines and a merge copy that stays incomplete are reported as status 1,
    and a refused cooperative launch is served by the single-pass kernel."""
    import shutil
    import subprocess
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.isfile(nvcc):
        pytest.skip("nvcc is not available on this machine")
    exe = str(tmp_path / "bounded_waits_test")
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O2", "-DTB200_TEST_HOOKS", "-DTB200_SPIN_LIMIT=65536",
                        "-I" + os.path.join(root, "include"), os.path.join(root, "tests", "cpp", "bounded_waits_test.cu"), "-o", exe],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "all checks passed" in r.stdout, r.stdout + r.stderr


def test_a_second_look_that_disagrees_is_reported(tb, tmp_path):
    """tests/cpp/predicate_twice_test.cu: the in-place partition looks at its items again before it stores over its input."""
    import shutil
    import subprocess
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.isfile(nvcc):
        pytest.skip("nvcc is not available on this machine")
    exe = str(tmp_path / "predicate_twice_test")
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O2", "-I" + os.path.join(root, "include"),
                        os.path.join(root, "tests", "cpp", "predicate_twice_test.cu"), "-o", exe], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "all checks passed" in r.stdout, r.stdout + r.stderr
