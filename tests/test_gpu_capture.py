"""Calls that only enqueue are captured into CUDA graphs and replayed on new contents of the same buffers, on every route
that a size takes: cooperative pipelines, the cluster sort, chains of overlapped launches."""
import numpy as np
import pytest
import torch

from thrust_b200 import datagen as dg
from gpu_util import dev, host

pytestmark = pytest.mark.gpu


def _captured(work):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        work()                                  # workspaces exist before the capture
    torch.cuda.current_stream().wait_stream(side)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        work()
    return g


@pytest.mark.parametrize("n", [1000, 50001, (1 << 20) + 3, (1 << 22) + 5])
def test_scan_and_sorts_replay(tb, port, n):
    x, keys, vals = dev(dg.scan_input_i32(n)), dev(dg.sort_keys_u32(n)), dev(np.arange(n, dtype=np.uint32))
    out = torch.empty_like(x)
    k, v, m = keys.clone(), vals.clone(), []

    def work():
        tb.inclusive_scan(x, out=out, sync=False)
        k.copy_(keys)
        v.copy_(vals)
        tb.sort_by_key(k, v, sync=False)
        m[:] = [tb.merge_by_key(k, k, v, v, sync=False)]

    g = _captured(work)
    for seed in (1, 2):
        h, hk = dg.scan_input_i32(n, seed), dg.rand64(seed, n).astype(np.uint32)
        x.copy_(dev(h))
        keys.copy_(dev(hk))
        g.replay()
        wk, wv = port.sort_by_key(hk, np.arange(n, dtype=np.uint32))
        assert np.array_equal(host(out), port.inclusive_scan(h))
        assert np.array_equal(host(k), wk) and np.array_equal(host(v), wv)
        mk, mv = port.merge_by_key(wk, wk, wv, wv)
        assert np.array_equal(host(m[0][0]), mk) and np.array_equal(host(m[0][1]), mv)
    del g
