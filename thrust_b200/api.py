"""Host-side mirror of the Thrust algorithms on the hot path, over the C ABI.

Function names, argument meaning and return conventions follow the reference's CUDA backend
(thrust/system/cuda/detail/{reduce,scan,sort,copy_if,partition,unique,reduce_by_key,merge}.h):
synchronous on return, results that are counts come back as Python ints, "end iterators" come
back as the output tensor sliced to its logical length.  Inputs are CUDA torch tensors; torch is
used only to own device memory and to name the stream.  Every call goes through
libthrust_b200.so; there is no fallback path.
"""
import ctypes as C
import struct
import threading

import numpy as np
import torch

from . import _lib

DTYPE_CODE = {
    torch.int8: 0, torch.uint8: 1, torch.int16: 2, torch.uint16: 3, torch.int32: 4,
    torch.uint32: 5, torch.int64: 6, torch.uint64: 7, torch.float32: 8, torch.float64: 9,
}
NP_OF = {
    torch.int8: np.int8, torch.uint8: np.uint8, torch.int16: np.int16, torch.uint16: np.uint16,
    torch.int32: np.int32, torch.uint32: np.uint32, torch.int64: np.int64, torch.uint64: np.uint64,
    torch.float32: np.float32, torch.float64: np.float64,
}
TORCH_OF = {np.dtype(v): k for k, v in NP_OF.items()}
OPS = {"plus": 0, "min": 1, "max": 2}
PREDS = {"mod_eq": 0, "lt": 1, "ge": 2, "ne": 3}


class Tb200Error(RuntimeError):
    """A C-ABI call returned a CUDA error, or a kernel reported a failed wait."""


def _check(rc, what):
    if rc != 0:
        raise Tb200Error("%s failed with cudaError %d" % (what, rc))


def _ptr(t):
    return None if t is None else t.data_ptr()


# the raw handle of a device's current stream, without building a torch.cuda.Stream around it where torch offers that
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda dev: torch.cuda.current_stream(dev).cuda_stream)


def _stream():
    return _raw_stream(torch.cuda.current_device())


def _require_cuda(*tensors):
    for t in tensors:
        if t is not None and (not t.is_cuda or not t.is_contiguous()):
            raise ValueError("thrust_b200 operates on contiguous CUDA tensors")


# the workspace header (ws_header in common.cuh): status, ticket, count, ..., and from byte 32 on room that a result may use
_HEADER = struct.Struct("<IIQ")
_HEADER_RESULT, _HEADER_BYTES = 32, 256


class _Kept:
    """One kept buffer: the tensor, its address and size as the C ABI takes them, its lock (re-entrant), and where its
    header is read to."""
    __slots__ = ("lock", "buf", "ptr", "size", "size_ref", "head")

    def __init__(self):
        self.lock = threading.RLock()
        self.head = C.create_string_buffer(_HEADER_BYTES)
        self.keep(None)

    def keep(self, buf):
        self.buf = buf
        self.ptr = None if buf is None else buf.data_ptr()
        self.size = C.c_size_t(0 if buf is None else buf.numel())
        self.size_ref = C.byref(self.size)


class _Workspaces:
    """Scratch buffers cached per (device, stream, call site) and grown on demand, standing in for
    the reference's per-call temporary_array (thrust/system/cuda/detail/reduce.h:959).

    Threads that share a stream share its buffers too, and a call's status, count or result lies in one until it
    is read back; a call therefore holds the buffer's lock from its first launch to that read-back."""

    def __init__(self):
        self._kept = {}

    @staticmethod
    def key(tag):
        """What the buffer of this call site on the current stream is kept under: (device, stream handle, tag)."""
        dev = torch.cuda.current_device()
        return dev, _raw_stream(dev), tag

    def at(self, key):
        return self._kept.get(key) or self._kept.setdefault(key, _Kept())

    def get(self, tag, nbytes, key=None):
        kept = self.at(key or self.key(tag))
        if kept.buf is None or kept.size.value < nbytes:
            kept.keep(torch.empty(max(int(nbytes), 256), dtype=torch.uint8, device="cuda"))
        return kept.buf

    def clear(self):
        for kept in list(self._kept.values()):
            with kept.lock:
                kept.keep(None)


workspaces = _Workspaces()


_TOO_SMALL = 1      # cudaErrorInvalidValue: the workspace is too small, or something else about the call is wrong


def _enqueue(key, kept, fn, args, result=None):
    """fn(*args, d_ws, &ws_bytes, stream) in the workspace kept under `key`, whose lock the caller holds; with `result`, an
    offset into the workspace, its address goes in front of d_ws.  The size is asked for only if there is no workspace yet
    or the call is refused, and the call made again only if the workspace was indeed too small (then nothing was
    launched: every entry point checks the size first)."""
    lib_fn = getattr(_lib.load(), fn)
    stream = key[1]
    rc = None
    if kept.ptr is not None:
        out = () if result is None else (kept.ptr + result,)
        rc = lib_fn(*args, *out, kept.ptr, kept.size_ref, stream)
        if rc != _TOO_SMALL:
            return _check(rc, fn)
    need = C.c_size_t(0)
    none = () if result is None else (None,)
    _check(lib_fn(*args, *none, None, C.byref(need), stream), fn + " (size query)")
    if rc is not None and kept.size.value >= need.value:
        _check(rc, fn)
    workspaces.get(key[2], need.value, key)
    out = () if result is None else (kept.ptr + result,)
    _check(lib_fn(*args, *out, kept.ptr, kept.size_ref, stream), fn)


def _enqueue_and_read(key, kept, what, fn, args, nbytes=_HEADER.size, result=None):
    """_enqueue, then the first `nbytes` of the header to kept.head once the stream has got there; returns the count.  The
    read is announced, so that the kernels can leave there what it fetches."""
    lib = _lib.load()
    if kept.ptr is None:      # the first call makes the workspace
        _enqueue(key, kept, fn, args, result)
    else:
        announced = kept.ptr
        lib.tb200_workspace_watch(announced)
        try:
            _enqueue(key, kept, fn, args, result)
        except BaseException:
            lib.tb200_workspace_watch(None)
            raise
        if kept.ptr != announced:      # refused there, and made in a larger one
            lib.tb200_workspace_watch(None)
    return _read_header(lib, kept.ptr, what, key[1], kept.head, nbytes)


def _read_header(lib, ptr, what, stream, head, nbytes):
    """Waits for the stream and reads the first `nbytes` of the workspace's header to `head`; returns the count and raises if
    the kernels reported a wait that ran out or looks at a tile that disagree."""
    rc = lib.tb200_workspace_read(ptr, nbytes, head, stream)
    if rc != 0:
        _check(rc, what + " (result)")
    status, _, count = _HEADER.unpack_from(head)
    if status != 0:
        raise Tb200Error("%s: device reported status %d (%s)" % (what, status, "an inter-CTA wait ran out" if status == 1 else "two looks at a tile disagree"))
    return count


def _call_with_ws(tag, fn, *args):
    """Enqueues fn in the workspace of the call site; returns the workspace."""
    key = workspaces.key(tag)
    kept = workspaces.at(key)
    with kept.lock:
        _enqueue(key, kept, fn, args)
        return kept.buf


def _call_and_wait(tag, what, fn, *args, sync=True, key=None):
    """The same, then (sync) waits for the stream and checks the status.  Returns the number that the kernels of
    a selecting or counting call left in the header.  key: the workspace's, if the caller has it."""
    key = key or workspaces.key(tag)
    kept = workspaces.at(key)
    with kept.lock:
        return _enqueue_and_read(key, kept, what, fn, args) if sync else _enqueue(key, kept, fn, args)


def _sync_and_check(ws, what):
    _read_header(_lib.load(), ws.data_ptr(), what, _stream(), C.create_string_buffer(_HEADER.size), _HEADER.size)


# ------------------------------------------------------------------------------------- reduce
def reduce(x, init=None, op="plus", acc_dtype=None):
    """thrust::reduce(first, last, init, op): returns init (+) x[0] (+) ... as a numpy scalar of the
    accumulator type (the type of `init`; default: x's type and 0, as in reduce.h:1057-1067)."""
    _require_cuda(x)
    if acc_dtype is None:
        acc_dtype = x.dtype if init is None or not isinstance(init, np.generic) else TORCH_OF[np.dtype(init.dtype)]
    h_init = np.asarray(0 if init is None else init, dtype=NP_OF[acc_dtype])
    # the result lands in the workspace's header and comes back together with the status
    key = workspaces.key("reduce")
    args = (_ptr(x), x.numel(), DTYPE_CODE[x.dtype], DTYPE_CODE[acc_dtype], OPS[op], h_init.tobytes())
    kept = workspaces.at(key)
    with kept.lock:
        _enqueue_and_read(key, kept, "reduce", "tb200_reduce", args, _HEADER_RESULT + 8, _HEADER_RESULT)
        return np.frombuffer(kept.head, dtype=h_init.dtype, count=1, offset=_HEADER_RESULT)[0]


def reduce_to_device(x, init, op="plus", acc_dtype=None, out=None):
    """The same reduction with the result left in device memory (a 1-element tensor of the accumulator
    type) and nothing waited for: for callers that feed it to later work on the stream."""
    _require_cuda(x)
    acc_dtype = acc_dtype or x.dtype
    h_init = np.asarray(init, dtype=NP_OF[acc_dtype])
    out = torch.empty(1, dtype=acc_dtype, device=x.device) if out is None else out
    _call_with_ws("reduce", "tb200_reduce", _ptr(x), x.numel(), DTYPE_CODE[x.dtype], DTYPE_CODE[acc_dtype], OPS[op],
                  h_init.tobytes(), _ptr(out))
    return out


# ------------------------------------------------------------------------------------- scan
def inclusive_scan(x, out=None, op="plus", init=None, sync=True):
    """thrust::inclusive_scan(first, last, result, op); out may be x (in place).  Returns out.
    `init`, if given, is combined in front of the first element (the carry of a sharded scan): a
    host scalar, or a 1-element CUDA tensor of x's type that earlier work on the stream fills in."""
    _require_cuda(x, out)
    out = torch.empty_like(x) if out is None else out
    if isinstance(init, torch.Tensor):
        _call_and_wait("scan", "inclusive_scan", "tb200_inclusive_scan_dinit", _ptr(x), _ptr(out), x.numel(), DTYPE_CODE[x.dtype], OPS[op],
                       _ptr(init), sync=sync)
    else:
        h_init = None if init is None else np.asarray(init, dtype=NP_OF[x.dtype])
        _call_and_wait("scan", "inclusive_scan", "tb200_inclusive_scan", _ptr(x), _ptr(out), x.numel(), DTYPE_CODE[x.dtype], OPS[op],
                       None if h_init is None else h_init.tobytes(), sync=sync)
    return out


def exclusive_scan(x, init=0, out=None, op="plus", sync=True):
    """thrust::exclusive_scan(first, last, result, init, op); init as for inclusive_scan."""
    _require_cuda(x, out)
    out = torch.empty_like(x) if out is None else out
    if isinstance(init, torch.Tensor):
        _call_and_wait("scan", "exclusive_scan", "tb200_exclusive_scan_dinit", _ptr(x), _ptr(out), x.numel(), DTYPE_CODE[x.dtype], OPS[op],
                       _ptr(init), sync=sync)
    else:
        h_init = np.asarray(init, dtype=NP_OF[x.dtype])
        _call_and_wait("scan", "exclusive_scan", "tb200_exclusive_scan", _ptr(x), _ptr(out), x.numel(), DTYPE_CODE[x.dtype], OPS[op],
                       h_init.tobytes(), sync=sync)
    return out


# ------------------------------------------------------------------------------------- sort
def _sort_impl(keys, vals, descending, begin_bit, end_bit, sync=True):
    _require_cuda(keys, vals)
    if vals is not None and vals.numel() != keys.numel():
        raise ValueError("keys and values differ in length")
    n = keys.numel()
    vb = 0 if vals is None else vals.element_size()
    end_bit = 8 * keys.element_size() if end_bit is None else end_bit
    key = workspaces.key("sort_keys_alt")
    with workspaces.at(key).lock:
        kalt = workspaces.get("sort_keys_alt", n * keys.element_size(), key)
        valt = None if vals is None else workspaces.get("sort_vals_alt", n * vb, key[:2] + ("sort_vals_alt",))
        _call_and_wait("sort", "sort", "tb200_sort_by_key", _ptr(keys), _ptr(kalt), _ptr(vals), _ptr(valt), n,
                       DTYPE_CODE[keys.dtype], vb, int(descending), begin_bit, end_bit, sync=sync, key=key[:2] + ("sort",))


def sort(keys, descending=False, sync=True):
    """thrust::sort / thrust::stable_sort(first, last[, greater]) in place.  sync=False only
    enqueues the work (for callers that chain several calls on one stream)."""
    _sort_impl(keys, None, descending, 0, None, sync)
    return keys


stable_sort = sort


def sort_by_key(keys, vals, descending=False, begin_bit=0, end_bit=None, sync=True):
    """thrust::sort_by_key / stable_sort_by_key(keys_first, keys_last, values_first[, greater]) in
    place; stable."""
    _sort_impl(keys, vals, descending, begin_bit, end_bit, sync)
    return keys, vals


stable_sort_by_key = sort_by_key

_side_streams = {}


def sort_by_key_host(h_keys, h_vals, h_keys_out=None, h_vals_out=None, descending=False):
    """thrust::sort_by_key for keys and values that start and end in (pinned) host memory: the call
    a host-side caller makes when the data does not live on the device.  The keys go up first and are
    sorted together with their positions while the values are still on their way up on a second
    stream; the sorted keys then travel back down while the values finish arriving (PCIe carries
    both directions at once), the values are permuted by the sorted positions (tb200_gather) and
    follow.  The result equals sort_by_key's on the same data (the sort is stable).  h_*_out default
    to the inputs (in place).  Returns (h_keys_out, h_vals_out) after synchronising."""
    if h_keys.is_cuda or h_vals.is_cuda:
        raise ValueError("sort_by_key_host takes host tensors; device tensors go to sort_by_key")
    n = h_keys.numel()
    if h_vals.numel() != n or h_vals.element_size() not in (4, 8) or n > 0xFFFFFFFF:
        raise ValueError("need one 4- or 8-byte value per key and at most 2^32 - 1 pairs")
    h_keys_out = h_keys if h_keys_out is None else h_keys_out
    h_vals_out = h_vals if h_vals_out is None else h_vals_out
    if n == 0:
        return h_keys_out, h_vals_out
    lib = _lib.load()
    dev = torch.cuda.current_device()
    main = torch.cuda.current_stream()
    side = _side_streams.get(dev)
    if side is None:
        side = _side_streams[dev] = torch.cuda.Stream()
    vb = h_vals.element_size()
    d_keys = workspaces.get("host_sort_keys", n * h_keys.element_size()).view(h_keys.dtype)[:n]
    d_pos = workspaces.get("host_sort_pos", n * 4).view(torch.int32)[:n]
    d_vals = workspaces.get("host_sort_vals", n * vb).view(h_vals.dtype)[:n]
    d_vals_out = workspaces.get("host_sort_vals_out", n * vb).view(h_vals.dtype)[:n]
    d_keys.copy_(h_keys.view(-1), non_blocking=True)
    keys_up = torch.cuda.Event()
    keys_up.record(main)
    side.wait_stream(main)                              # the value buffer may still be read by an earlier call's gather
    with torch.cuda.stream(side):
        side.wait_event(keys_up)                        # keys first: the sort can start while the values follow
        d_vals.copy_(h_vals.view(-1), non_blocking=True)
        vals_up = torch.cuda.Event()
        vals_up.record(side)
    _check(lib.tb200_sequence_u32(_ptr(d_pos), n, _stream()), "tb200_sequence_u32")
    sort_by_key(d_keys, d_pos, descending, sync=False)
    h_keys_out.view(-1).copy_(d_keys, non_blocking=True)
    main.wait_event(vals_up)
    _check(lib.tb200_gather(_ptr(d_vals), _ptr(d_pos), _ptr(d_vals_out), n, vb, _stream()), "tb200_gather")
    h_vals_out.view(-1).copy_(d_vals_out, non_blocking=True)
    _sync_and_check(workspaces.get("sort", 1), "sort_by_key_host")      # waits for the stream
    return h_keys_out, h_vals_out


# ------------------------------------------------------------------------------------- compaction
def copy_if(x, pred, a=0, b=0, stencil=None, out=None):
    """thrust::copy_if(first, last, [stencil,] result, pred): returns out[:count] (stable)."""
    _require_cuda(x, stencil, out)
    out = torch.empty_like(x) if out is None else out
    count = _call_and_wait("select", "copy_if", "tb200_copy_if", _ptr(x), _ptr(stencil), _ptr(out), x.numel(), DTYPE_CODE[x.dtype],
                           0 if stencil is None else DTYPE_CODE[stencil.dtype], PREDS[pred], a, b, None)
    return out[:count]


def partition_copy(x, pred, a=0, b=0, stencil=None):
    """thrust::stable_partition_copy: returns (selected, rejected), both in input order."""
    _require_cuda(x, stencil)
    out_t, out_f = torch.empty_like(x), torch.empty_like(x)
    k = _call_and_wait("select", "partition_copy", "tb200_partition_copy", _ptr(x), _ptr(stencil), _ptr(out_t), _ptr(out_f), x.numel(),
                       DTYPE_CODE[x.dtype], 0 if stencil is None else DTYPE_CODE[stencil.dtype], PREDS[pred], a, b, None)
    return out_t[:k], out_f[:x.numel() - k]


stable_partition_copy = partition_copy


def partition(x, pred, a=0, b=0):
    """thrust::partition / thrust::stable_partition in place; returns the split point."""
    _require_cuda(x)
    return _call_and_wait("partition", "partition", "tb200_partition", _ptr(x), x.numel(), DTYPE_CODE[x.dtype], PREDS[pred], a, b, None)


stable_partition = partition


def unique_copy(x, out=None):
    """thrust::unique_copy(first, last, result): returns out[:count]."""
    _require_cuda(x, out)
    out = torch.empty_like(x) if out is None else out
    count = _call_and_wait("select", "unique_copy", "tb200_unique_copy", _ptr(x), _ptr(out), x.numel(), DTYPE_CODE[x.dtype], None)
    return out[:count]


def unique(x):
    """thrust::unique(first, last) in place: returns x[:count]."""
    return unique_copy(x, out=x)


def reduce_by_key(keys, vals, op="plus"):
    """thrust::reduce_by_key(keys_first, keys_last, values_first, keys_out, values_out, equal_to, op):
    returns (keys_out[:runs], values_out[:runs])."""
    _require_cuda(keys, vals)
    ko, vo = torch.empty_like(keys), torch.empty_like(vals)
    k = _call_and_wait("rbk", "reduce_by_key", "tb200_reduce_by_key", _ptr(keys), _ptr(vals), _ptr(ko), _ptr(vo), keys.numel(),
                       DTYPE_CODE[keys.dtype], DTYPE_CODE[vals.dtype], OPS[op], None)
    return ko[:k], vo[:k]


def inclusive_scan_by_key(keys, vals, out=None, op="plus"):
    """thrust::inclusive_scan_by_key(keys_first, keys_last, values_first, result, equal_to, op)."""
    _require_cuda(keys, vals, out)
    out = torch.empty_like(vals) if out is None else out
    _call_and_wait("rbk", "inclusive_scan_by_key", "tb200_scan_by_key", _ptr(keys), _ptr(vals), _ptr(out), keys.numel(), DTYPE_CODE[keys.dtype],
                   DTYPE_CODE[vals.dtype], OPS[op], 0, None)
    return out


def exclusive_scan_by_key(keys, vals, init=0, out=None, op="plus"):
    """thrust::exclusive_scan_by_key(keys_first, keys_last, values_first, result, init, equal_to, op)."""
    _require_cuda(keys, vals, out)
    out = torch.empty_like(vals) if out is None else out
    h_init = np.asarray(init, dtype=NP_OF[vals.dtype])
    _call_and_wait("rbk", "exclusive_scan_by_key", "tb200_scan_by_key", _ptr(keys), _ptr(vals), _ptr(out), keys.numel(), DTYPE_CODE[keys.dtype],
                   DTYPE_CODE[vals.dtype], OPS[op], 1, h_init.tobytes())
    return out


def unique_by_key_copy(keys, vals, keys_out=None, vals_out=None):
    """thrust::unique_by_key_copy: returns (keys_out[:runs], vals_out[:runs])."""
    _require_cuda(keys, vals, keys_out, vals_out)
    ko = torch.empty_like(keys) if keys_out is None else keys_out
    vo = torch.empty_like(vals) if vals_out is None else vals_out
    k = _call_and_wait("rbk", "unique_by_key_copy", "tb200_unique_by_key_copy", _ptr(keys), _ptr(vals), _ptr(ko), _ptr(vo), keys.numel(),
                       DTYPE_CODE[keys.dtype], vals.element_size(), None)
    return ko[:k], vo[:k]


def unique_by_key(keys, vals):
    """thrust::unique_by_key in place: returns (keys[:runs], vals[:runs])."""
    return unique_by_key_copy(keys, vals, keys, vals)


# ------------------------------------------------------------------------------------- extrema
def _extrema(fn, x, words):
    _require_cuda(x)
    idx = torch.zeros(words, dtype=torch.int64, device="cuda")
    _call_and_wait("reduce", fn, fn, _ptr(x), x.numel(), DTYPE_CODE[x.dtype], _ptr(idx))
    return [int(v) for v in idx.cpu().tolist()]


def min_element(x):
    """thrust::min_element(first, last): position of the first smallest element (0 when empty)."""
    return _extrema("tb200_min_element", x, 1)[0]


def max_element(x):
    """thrust::max_element(first, last): position of the first largest element (0 when empty)."""
    return _extrema("tb200_max_element", x, 1)[0]


def minmax_element(x):
    """thrust::minmax_element(first, last): (position of the first smallest, of the first largest)."""
    lo, hi = _extrema("tb200_minmax_element", x, 2)
    return lo, hi


# ------------------------------------------------------------------------------------- merge
def merge_by_key(keys_a, keys_b, vals_a=None, vals_b=None, descending=False, sync=True):
    """thrust::merge_by_key(A, B, payload A, payload B, keys_out, payload_out[, greater]); with no
    payloads it is thrust::merge.  Returns (keys_out, payload_out or None)."""
    _require_cuda(keys_a, keys_b, vals_a, vals_b)
    if keys_a.dtype != keys_b.dtype:
        raise ValueError("key types differ")
    na, nb = keys_a.numel(), keys_b.numel()
    ko = torch.empty(na + nb, dtype=keys_a.dtype, device=keys_a.device)
    vo = None if vals_a is None else torch.empty(na + nb, dtype=vals_a.dtype, device=keys_a.device)
    vb = 0 if vals_a is None else vals_a.element_size()
    _call_and_wait("merge", "merge_by_key", "tb200_merge_by_key", _ptr(keys_a), _ptr(vals_a), na, _ptr(keys_b), _ptr(vals_b), nb, _ptr(ko),
                   _ptr(vo), DTYPE_CODE[keys_a.dtype], vb, int(descending), sync=sync)
    return ko, vo


def merge(a, b, descending=False):
    """thrust::merge(A, B, out[, greater])."""
    return merge_by_key(a, b, None, None, descending)[0]


SET_OPS = {"union": 0, "intersection": 1, "difference": 2, "symmetric_difference": 3}


def set_operation(op, keys_a, keys_b, vals_a=None, vals_b=None, descending=False):
    """thrust::set_union / set_intersection / set_difference / set_symmetric_difference (op names
    as in SET_OPS) of two sorted ranges, and their _by_key forms when vals_a is given (vals_b for the
    union and the symmetric difference, whose results also take items from B).  Returns
    (keys_out, vals_out or None) cut to the result's length."""
    _require_cuda(keys_a, keys_b, vals_a, vals_b)
    if keys_a.dtype != keys_b.dtype:
        raise ValueError("key types differ")
    code = SET_OPS[op]
    na, nb = keys_a.numel(), keys_b.numel()
    cap = {0: na + nb, 1: min(na, nb), 2: na, 3: na + nb}[code]
    ko = torch.empty(cap, dtype=keys_a.dtype, device=keys_a.device)
    vo = None if vals_a is None else torch.empty(cap, dtype=vals_a.dtype, device=keys_a.device)
    vb = 0 if vals_a is None else vals_a.element_size()
    m = _call_and_wait("setop", "set_" + op, "tb200_set_operation", code, _ptr(keys_a), na, _ptr(keys_b), nb, _ptr(vals_a), _ptr(vals_b),
                       _ptr(ko), _ptr(vo), DTYPE_CODE[keys_a.dtype], vb, int(descending), None)
    return ko[:m], (None if vo is None else vo[:m])


def merge_sort_by_key(keys, vals=None, descending=False):
    """The comparison-sort route of thrust::stable_sort(_by_key): stable merge sort in place."""
    _require_cuda(keys, vals)
    n = keys.numel()
    vb = 0 if vals is None else vals.element_size()
    key = workspaces.key("sort_keys_alt")
    with workspaces.at(key).lock:
        kalt = workspaces.get("sort_keys_alt", n * keys.element_size(), key)
        valt = None if vals is None else workspaces.get("sort_vals_alt", n * vb, key[:2] + ("sort_vals_alt",))
        _call_and_wait("merge_sort", "merge_sort_by_key", "tb200_merge_sort_by_key", _ptr(keys), _ptr(kalt), _ptr(vals), _ptr(valt), n,
                       DTYPE_CODE[keys.dtype], vb, int(descending), key=key[:2] + ("merge_sort",))
    return keys, vals


def stable_sort_zip_by_first(keys, vals, method="merge"):
    """thrust::stable_sort(zip(keys, vals), comp) with comp ordering on get<0> alone, in place.
    method "merge" follows the reference's comparator route (merge sort); "radix" uses the fact
    that the comparator is a plain less on an arithmetic key and takes the radix path."""
    if method == "radix":
        return sort_by_key(keys, vals)
    return merge_sort_by_key(keys, vals)
