"""Host threads that share a stream, and with it the kept workspaces, each get their own results."""
import threading

import numpy as np
import pytest

from thrust_b200 import datagen as dg
from gpu_util import dev, host

pytestmark = pytest.mark.gpu


def test_two_threads_on_the_default_stream(tb, port):
    """reduce, copy_if, partition_copy, sort and reduce_by_key of different inputs from two threads: sums, counts and
    contents are each thread's own in every one of the passes."""
    sizes = (30011, 70001)
    wrong = []

    def work(i):
        x = dg.compaction_input(sizes[i]) + i
        k = dg.run_keys(sizes[i])
        xd, kd = dev(x), dev(k)
        total, kept, (rk, rv) = x.astype(np.int64).sum(), port.copy_if(x, "mod_eq", 3, 1), port.reduce_by_key(k, k)
        for _ in range(100):
            if tb.reduce(xd, np.int64(0)) != total:
                wrong.append("reduce")
            c = tb.copy_if(xd, "mod_eq", 3, 1)
            if c.numel() != kept.size or not np.array_equal(host(c), kept):
                wrong.append("copy_if")
            sel, rej = tb.partition_copy(xd, "mod_eq", 3, 1)
            if sel.numel() != kept.size or rej.numel() != x.size - kept.size:
                wrong.append("partition_copy")
            gk, gv = tb.reduce_by_key(kd, kd)
            if gk.numel() != rk.size or not np.array_equal(host(gv), rv):
                wrong.append("reduce_by_key")
            s = xd.clone()
            tb.sort(s)
            if not np.array_equal(host(s), np.sort(x)):
                wrong.append("sort")

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, sorted(set(wrong))
