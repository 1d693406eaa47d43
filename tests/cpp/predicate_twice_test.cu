// The in-place partition stores over its own input, so what a tile stores is looked at again before it is stored: a second look that
// disagrees with the first is status 2.  Shown with a predicate that answers true the first time it sees an item and false after that.
#include <cstdio>
#include <vector>

#include "thrust_b200/select.cuh"

constexpr size_t N = ((size_t)1 << 21) + 4099;

struct true_once {
  unsigned* calls;
  __device__ bool operator()(int x) const { return (unsigned)x < N && atomicAdd(calls + x, 1u) == 0; }
};

int main() {
  std::vector<int> h(N);
  for (size_t i = 0; i < N; ++i) h[i] = (int)i;
  int *data, *scratch;
  unsigned* calls;
  void* ws;
  tb200::ws_header head;
  bool ok = cudaMalloc(&data, 4 * N) == cudaSuccess && cudaMalloc(&scratch, 4 * N) == cudaSuccess && cudaMalloc(&calls, 4 * N) == cudaSuccess &&
            cudaMalloc(&ws, 64 << 20) == cudaSuccess && cudaMemcpy(data, h.data(), 4 * N, cudaMemcpyHostToDevice) == cudaSuccess && cudaMemset(calls, 0, 4 * N) == cudaSuccess;
  ok = ok && tb200::partition_inplace_async(data, scratch, N, true_once{calls}, nullptr, ws, 0) == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
  ok = ok && cudaMemcpy(&head, ws, sizeof(head), cudaMemcpyDeviceToHost) == cudaSuccess;
  std::printf("status %u\n", head.error);
  ok = ok && head.error == tb200::ERR_INCONSISTENT;
  std::printf(ok ? "predicate_twice_test: all checks passed\n" : "predicate_twice_test: FAILED\n");
  return ok ? 0 : 1;
}
