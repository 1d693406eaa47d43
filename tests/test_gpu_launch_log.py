"""THRUST_B200_LOG=1: one line per dominant launch, whichever route a call takes."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import torch, thrust_b200 as tb
x = torch.arange(1 << 19, dtype=torch.int32, device="cuda")
%s
"""


@pytest.mark.parametrize("call,kernels", [
    ("tb.sort(x[:5000].clone())", ["cluster_sort_kernel"]),
    ("tb.sort(x.clone())", ["radix_hist_kernel", "onesweep_kernel"]),
    ("tb.merge(x, x)", ["merge_slices_kernel"]),
    ("tb.merge_sort_by_key(x.clone())", ["block_sort_kernel", "merge_slices_kernel"]),
    ("tb.partition(x.clone(), 'lt', 77)", ["select_pipe_kernel", "partition_rejects_kernel"]),
    ("tb.reduce_by_key(x, x)", ["rbk_pipe_kernel"]),
])
def test_every_route_logs_its_kernels(tb, call, kernels):
    r = subprocess.run([sys.executable, "-c", PROGRAM % call], capture_output=True, text=True, cwd=ROOT, env=dict(os.environ, THRUST_B200_LOG="1"), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    for k in kernels:
        assert any(k + "<<<" in line and "cudaSuccess" in line for line in r.stderr.splitlines()), (k, r.stderr[-2000:])
