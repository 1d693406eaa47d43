"""Kernels compiled (not run) at the element sizes where their static shared memory comes closest to its 48 KB."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "thrust_b200/merge.cuh"
template <int WORDS> struct key { int w[WORDS]; };
struct by_first_word { template <class K> __host__ __device__ bool operator()(const K& a, const K& b) const { return a.w[0] < b.w[0]; } };
template <int WORDS> cudaError_t sort(void* p, size_t n) {
  using K = key<WORDS>;
  return tb200::merge_sort_async<K, unsigned, false>((K*)p, (K*)p + n, (unsigned*)nullptr, (unsigned*)nullptr, n, by_first_word(), p, 0);
}
cudaError_t all(void* p, size_t n) {
  cudaError_t e = cudaSuccess;
  %s
  return e;
}
"""


@pytest.mark.parametrize("words", [[4, 5, 6], [9, 10, 42]])
def test_comparator_sort_of_any_key_size_compiles(tmp_path, words):
    """16-, 20- and 24-byte keys lie around the size at which the block sort's padded tile no longer fits, 36 and 40
    around the next smaller tile, 168 is the largest."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.isfile(nvcc):
        pytest.skip("nvcc is not available on this machine")
    src = tmp_path / "sort_sizes.cu"
    src.write_text(SOURCE % "\n  ".join("if (e == cudaSuccess) e = sort<%d>(p, n);" % w for w in words))
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + os.path.join(ROOT, "include"), "-c", str(src),
                        "-o", str(tmp_path / "sort_sizes.o")], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr


def test_comparator_sort_of_the_largest_keys_compiles(tmp_path):
    """188 bytes is the largest key of whole words."""
    test_comparator_sort_of_any_key_size_compiles(tmp_path, [46, 47])


def test_merge_tiles_stay_inside_their_inputs(tmp_path):
    """Sorted keys with NaNs strewn in are no ordered ranges: tiles whose two splits disagree are refused, all others have
    slices inside A and B (tests/cpp/merge_slices_host.cu, host code only)."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.isfile(nvcc):
        pytest.skip("nvcc is not available on this machine")
    exe = str(tmp_path / "merge_slices_host")
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "tests", "cpp", "merge_slices_host.cu"), "-o", exe], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("tunables", [[], ["-DTB200_RBK_IPT4=255"]])
def test_workspaces_hold_every_route(tmp_path, tunables):
    """Also where the single-pass kernel's tiles are tuned larger than the pipeline's (tests/cpp/workspace_bounds_host.cu, host
    code only)."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.isfile(nvcc):
        pytest.skip("nvcc is not available on this machine")
    exe = str(tmp_path / "workspace_bounds_host")
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + os.path.join(ROOT, "include"), *tunables,
                        os.path.join(ROOT, "tests", "cpp", "workspace_bounds_host.cu"), "-o", exe], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
