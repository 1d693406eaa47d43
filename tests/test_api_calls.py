"""The Python layer's way through a call -- size query, workspace, launch, read-back -- with a stand-in for the library
on the CPU, so that what another thread or an error code does in between can be arranged."""
import ctypes as C
import struct
import threading

import numpy as np
import pytest
import torch

from thrust_b200 import _lib, api

NEED = 512


class FakeLibrary:
    """tb200_reduce (int64 sums) and tb200_copy_if (x != a) on host memory, with the C ABI's workspace rules."""

    def __init__(self):
        self.between = lambda: None       # what happens between a call's launch and its read-back
        self.launches = []
        self.result = 0                   # what the next calls return once they are past the size check
        self.watched = []                 # what was announced, in order

    def _gate(self, d_ws, size):
        if d_ws is None:
            size._obj.value = NEED
            return 0
        return 1 if size._obj.value < NEED else None

    def _launched(self, name):
        self.launches.append(name)
        if self.result == 0:
            self.between()
        return self.result

    def tb200_reduce(self, x, n, in_t, acc_t, op, h_init, d_out, d_ws, size, stream):
        rc = self._gate(d_ws, size)
        if rc is not None:
            return rc
        C.memset(d_ws, 0, 256)
        C.memmove(d_out, struct.pack("<q", int(np.ctypeslib.as_array(C.cast(x, C.POINTER(C.c_int64)), (n,)).sum())), 8)
        return self._launched("reduce")

    def tb200_copy_if(self, x, stencil, out, n, t, stencil_t, pred, a, b, d_count, d_ws, size, stream):
        rc = self._gate(d_ws, size)
        if rc is not None:
            return rc
        h = np.ctypeslib.as_array(C.cast(x, C.POINTER(C.c_int64)), (n,))
        kept = np.ascontiguousarray(h[h != a])
        C.memmove(out, kept.ctypes.data, kept.nbytes)
        C.memmove(d_ws, struct.pack("<IIQ", 0, 0, kept.size), 16)
        return self._launched("copy_if")

    def tb200_workspace_watch(self, d_ws):
        self.watched.append(d_ws)
        return 0

    def tb200_workspace_read(self, d_ws, nbytes, dst, stream):
        C.memmove(dst, d_ws, nbytes)
        return 0


@pytest.fixture
def fake(monkeypatch):
    lib = FakeLibrary()
    monkeypatch.setattr(_lib, "_lib", lib)
    monkeypatch.setattr(api, "_require_cuda", lambda *t: None)
    monkeypatch.setattr(api, "_raw_stream", lambda dev: 0)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, device=None, **k: empty(*a, **k))
    monkeypatch.setattr(api, "workspaces", type(api.workspaces)())
    return lib


@pytest.mark.parametrize("name", ["reduce", "copy_if"])
def test_threads_on_one_stream_get_their_own_answers(fake, name):
    """Each call gives the other thread 0.2 s to launch in the workspace they share before it is read back."""
    met = threading.Barrier(2)

    def let_the_other_in():
        try:
            met.wait(timeout=0.2)
        except threading.BrokenBarrierError:
            pass

    fake.between = let_the_other_in
    got = [None, None]

    def work(i):
        x = torch.arange(10 * (i + 1), dtype=torch.int64)
        got[i] = int(api.reduce(x)) if name == "reduce" else api.copy_if(x, "ne", 3).numel()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == ([45, 190] if name == "reduce" else [9, 19])


@pytest.mark.parametrize("name", ["reduce", "copy_if"])
def test_a_refused_call_is_made_again_only_for_its_size(fake, name):
    """Error 1 from behind the size check is an error of the call, which may have launched something: raised, not retried.
    A workspace that is too small is replaced and the call made once more."""
    x = torch.arange(10, dtype=torch.int64)
    call = (lambda: api.reduce(x)) if name == "reduce" else (lambda: api.copy_if(x, "ne", 3))
    call()
    assert fake.launches == [name]
    fake.result = 1
    with pytest.raises(api.Tb200Error, match="cudaError 1"):
        call()
    assert fake.launches == [name] * 2
    fake.result = 0
    key = api.workspaces.key("reduce" if name == "reduce" else "select")
    api.workspaces.at(key).keep(torch.empty(NEED - 1, dtype=torch.uint8))
    call()
    assert fake.launches == [name] * 3 and api.workspaces.at(key).buf.numel() == NEED


@pytest.mark.parametrize("name", ["reduce", "copy_if"])
def test_a_failed_call_is_no_longer_announced(fake, name):
    x = torch.arange(10, dtype=torch.int64)
    call = (lambda: api.reduce(x)) if name == "reduce" else (lambda: api.copy_if(x, "ne", 3))
    call()
    call()
    kept = api.workspaces.at(api.workspaces.key("reduce" if name == "reduce" else "select"))
    assert fake.watched == [kept.ptr]              # the first call has made its workspace
    fake.result = 700
    with pytest.raises(api.Tb200Error):
        call()
    assert fake.watched == [kept.ptr, kept.ptr, None]


def test_a_workspace_that_was_replaced_is_no_longer_announced(fake):
    """Its memory may become another call's."""
    x = torch.arange(10, dtype=torch.int64)
    api.reduce(x)
    kept = api.workspaces.at(api.workspaces.key("reduce"))
    kept.keep(torch.empty(NEED - 1, dtype=torch.uint8))
    small = kept.ptr
    assert int(api.reduce(x)) == 45
    assert fake.watched == [small, None]
