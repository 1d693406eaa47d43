// A meeting of the grid sort that one CTA never comes to: the others' bounded waits run out, the kernel returns with status 1 and the
// context stays usable; the next call on the same workspace sorts.  Built with -DTB200_TEST_HOOKS and a short TB200_SPIN_LIMIT.
#include <stdio.h>
#include <algorithm>
#include <vector>
#include "thrust_b200/radix_sort.cuh"

int main() {
  const size_t n = 100003;
  std::vector<uint32_t> h(n);
  for (size_t i = 0; i < n; ++i) h[i] = (uint32_t)(i * 2654435761u);
  uint32_t *k, *alt;
  void* ws;
  const size_t bytes = tb200::radix_workspace_bytes<4, 0>(n);
  if (cudaMalloc(&k, n * 4) || cudaMalloc(&alt, n * 4) || cudaMalloc(&ws, bytes)) return 1;
  for (unsigned withheld : {1u, 0u}) {
    tb200::test_hook_flags() = withheld;
    cudaMemcpy(k, h.data(), n * 4, cudaMemcpyHostToDevice);
    const cudaError_t e = tb200::radix_sort_async<uint32_t, uint32_t, false>(k, alt, nullptr, nullptr, n, tb200::key_coding{tb200::KEY_UNSIGNED, 0}, 0, 32, ws, 0);
    unsigned status = 77;
    if (e != cudaSuccess || cudaMemcpy(&status, ws, 4, cudaMemcpyDeviceToHost) != cudaSuccess) { printf("launch or kernel failed\n"); return 1; }
    if (status != withheld) { printf("withheld %u: status %u\n", withheld, status); return 1; }
  }
  std::vector<uint32_t> got(n);
  cudaMemcpy(got.data(), k, n * 4, cudaMemcpyDeviceToHost);
  std::sort(h.begin(), h.end());
  if (got != h) { printf("not sorted\n"); return 1; }
  printf("all checks passed\n");
  return 0;
}
