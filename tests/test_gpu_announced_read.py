"""tb200_workspace_watch: an announced call reports to pinned memory, and whatever is done between it and its read, every workspace's
header answers for that workspace's last call."""
import ctypes as C
import struct
import threading

import numpy as np
import pytest

from thrust_b200 import _lib

pytestmark = pytest.mark.gpu
I32, I64, PLUS, RESULT = 4, 6, 0, 32


class Workspace:
    def __init__(self, lib=None):
        import torch
        self.lib = lib or _lib.load()
        self.size = C.c_size_t(0)
        assert self.lib.tb200_reduce(None, 8, I32, I64, PLUS, None, None, None, C.byref(self.size), None) == 0
        self.buf = torch.zeros(max(self.size.value, 1 << 20), dtype=torch.uint8, device="cuda")
        self.size = C.c_size_t(self.buf.numel())
        self.at = self.buf.data_ptr()

    def watch(self):
        assert self.lib.tb200_workspace_watch(self.at) == 0

    def reduce(self, x, stream=None):
        assert self.lib.tb200_reduce(x.data_ptr(), x.numel(), I32, I64, PLUS, struct.pack("<q", 0), self.at + RESULT, self.at, C.byref(self.size), stream) == 0

    def read(self, nbytes=RESULT + 8):
        head = C.create_string_buffer(nbytes)
        assert self.lib.tb200_workspace_read(self.at, nbytes, head, None) == 0
        assert struct.unpack_from("<I", head)[0] == 0
        return head.raw

    def result(self):
        return struct.unpack_from("<q", self.read(), RESULT)[0]

    def in_header(self):
        """What lies on the device."""
        return struct.unpack("<q", bytes(self.buf[RESULT:RESULT + 8].cpu().numpy()))[0]


@pytest.fixture
def ones(tb):
    import torch
    return lambda n: torch.ones(n, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("n", [1000, 300000])       # one cluster; partials and the last CTA
def test_another_workspace_is_read_in_between(ones, n):
    a, b = Workspace(), Workspace()
    b.reduce(ones(77))
    a.watch()
    a.reduce(ones(n))
    assert b.result() == 77
    assert a.result() == n
    assert (a.result(), b.result()) == (n, 77)      # read again, no longer announced


@pytest.mark.parametrize("n", [1000, 300000])
def test_an_announcement_withdrawn_behind_its_call(ones, n):
    a = Workspace()
    for i in range(20):                             # more often than blocks are put aside for
        a.watch()
        a.reduce(ones(n + i))
        assert a.lib.tb200_workspace_watch(None) == 0
        assert a.result() == n + i
    a.watch()
    a.reduce(ones(5))
    assert a.result() == 5


def test_only_the_next_call_is_announced(ones):
    a = Workspace()
    a.watch()
    a.reduce(ones(1000))
    a.reduce(ones(2000))
    assert a.in_header() == 2000
    assert a.result() == 2000


def test_a_captured_call_reports_to_its_workspace(ones):
    import torch
    a, x = Workspace(), ones(1000)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        a.reduce(x, side.cuda_stream)
    torch.cuda.synchronize()
    a.buf[:256].zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    a.watch()
    with torch.cuda.graph(graph, stream=side):
        a.reduce(x, side.cuda_stream)
    assert a.lib.tb200_workspace_watch(None) == 0
    x.fill_(3)
    graph.replay()
    torch.cuda.synchronize()
    assert a.in_header() == 3000
    assert a.result() == 3000


def test_a_callers_own_bytes_of_the_header(ones):
    """Bytes 32-255 are the caller's once a call has been enqueued; a read of the whole header finds them."""
    import torch
    a = Workspace()
    a.watch()
    a.reduce(ones(1000))
    a.buf[64:72] = torch.arange(8, dtype=torch.uint8, device="cuda")
    head = a.read(256)
    assert struct.unpack_from("<q", head, RESULT)[0] == 1000 and head[64:72] == bytes(range(8))


def test_a_thread_that_never_reads(ones):
    import torch
    a, x = Workspace(), ones(300000)

    def work():
        a.watch()
        a.reduce(x)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert a.in_header() == 300000


def test_status_of_an_announced_call(ones):
    """A wait that runs out (test build, tests/test_gpu_failure_path.py) is found by a status query before the read, by the read, and by a
    status query after it."""
    import os
    import torch
    from thrust_b200 import build
    if not os.path.isfile(build.SHORTWAIT_LIB):
        pytest.fail("%s is missing -- python -m thrust_b200.build makes it" % build.SHORTWAIT_LIB)
    short = _lib.load_partial(build.SHORTWAIT_LIB)
    short.tb200_test_hooks.argtypes = [C.c_uint]
    a = Workspace(short)
    n = 5 * 8192 + 123
    x = ones(n)
    out = torch.empty_like(x)
    assert short.tb200_test_hooks(1) == 0
    try:
        a.watch()
        assert short.tb200_inclusive_scan(x.data_ptr(), out.data_ptr(), n, I32, PLUS, None, a.at, C.byref(a.size), None) == 0
        status, head = C.c_uint(7), C.create_string_buffer(16)
        assert short.tb200_workspace_status(a.at, None, C.byref(status)) == 0 and status.value == 1
        assert short.tb200_workspace_read(a.at, 16, head, None) == 0 and struct.unpack_from("<I", head)[0] == 1
        assert short.tb200_workspace_status(a.at, None, C.byref(status)) == 0 and status.value == 1
    finally:
        assert short.tb200_test_hooks(0) == 0
    a.watch()
    assert short.tb200_inclusive_scan(x.data_ptr(), out.data_ptr(), n, I32, PLUS, None, a.at, C.byref(a.size), None) == 0
    assert short.tb200_workspace_read(a.at, 16, head, None) == 0 and struct.unpack_from("<I", head)[0] == 0
    assert np.array_equal(out.cpu().numpy(), np.arange(1, n + 1, dtype=np.int32))
