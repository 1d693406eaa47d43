// How a small reduction is spread over threads: behind an iterator every item has its own thread while there are threads for all of
// them, and a caller's operator is applied to one vector's items per thread, whichever route the call takes.
#include <cstdio>
#include <vector>

#include "thrust_b200/reduce.cuh"

constexpr unsigned THREADS = tb200::REDUCE_MAX_GRID * tb200::REDUCE_BLOCK;
__device__ __forceinline__ unsigned this_thread() { return blockIdx.x * tb200::REDUCE_BLOCK + threadIdx.x; }

struct counting_items {   // item i is i; counts the items that a thread asks for
  unsigned* asked;
  __device__ int operator[](size_t i) const { if (this_thread() < THREADS) atomicAdd(asked + this_thread(), 1u); return (int)i; }
};
struct counting_max {
  unsigned* applied;
  __device__ int operator()(int a, int b) const { if (this_thread() < THREADS) atomicAdd(applied + this_thread(), 1u); return a < b ? b : a; }
};

int main() {
  const size_t most = (size_t)tb200::current_device_info().sm_count * tb200::REDUCE_CTAS_PER_SM * tb200::REDUCE_BLOCK;
  const std::vector<size_t> sizes = {1, 255, 257, 1000, 4096, 4097, 30000, 65536, 131072, 131073};
  std::vector<int> h(sizes.back());
  for (size_t i = 0; i < h.size(); ++i) h[i] = (int)i;
  unsigned* counts;
  int *data, *out;
  void* ws = nullptr;
  bool ok = cudaMalloc(&counts, THREADS * 4) == cudaSuccess && cudaMalloc(&data, h.size() * 4) == cudaSuccess && cudaMalloc(&out, 4) == cudaSuccess &&
            cudaMalloc(&ws, tb200::reduce_workspace_bytes<int>()) == cudaSuccess && cudaMemcpy(data, h.data(), h.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess;
  std::vector<unsigned> seen(THREADS);
  auto check = [&](const char* what, size_t n, unsigned threads, unsigned limit, auto call) {
    int result = -1;
    const bool ran = cudaMemset(counts, 0, THREADS * 4) == cudaSuccess && call() == cudaSuccess && cudaMemcpy(&result, out, 4, cudaMemcpyDeviceToHost) == cudaSuccess &&
         cudaMemcpy(seen.data(), counts, THREADS * 4, cudaMemcpyDeviceToHost) == cudaSuccess;
    unsigned largest = 0, busy = 0;
    for (unsigned c : seen) { largest = c > largest ? c : largest; busy += c != 0; }
    const bool good = ran && result == (int)n - 1 && largest <= limit && busy >= threads;
    if (!good) std::printf("%s, %zu items: result %d, %u threads (at least %u), at most %u each (limit %u)\n", what, n, result, busy, threads, largest, limit);
    ok = ok && good;
  };
  for (size_t n : sizes) {
    if (!ws) break;
    const unsigned own = (unsigned)(n < most ? n : most);
    check("iterator", n, own, (unsigned)((n + most - 1) / most),
          [&] { return tb200::reduce_async(counting_items{counts}, n, 0, tb200::max_op(), out, ws, 0); });
    // per thread: 3 inside a vector and one for the ragged end, 5 + 3 up the warp and the CTA; the last to finish, or the cluster's first thread,
    // adds up at most 16 totals or ceil(592 / 256) partials, 5 + 3 levels of them, and init
    const size_t vectors = n / 4;
    check("operator", n, (unsigned)(vectors < most ? vectors : most), 4 + 8 + 16 + 8 + 1,
          [&] { return tb200::reduce_async((const int*)data, n, 0, counting_max{counts}, out, ws, 0); });
  }
  std::printf(ok ? "reduce_spread_test: all checks passed\n" : "reduce_spread_test: FAILED\n");
  return ok ? 0 : 1;
}
