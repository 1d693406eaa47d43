// Waits that run out: the pipelines of scan, compaction, in-place partition and reduce_by_key with tile 0's descriptor withheld, a merge
// whose tiles wait for bytes that nobody sends, and a pipeline launch that the device refuses.  Compiled with
// -DTB200_TEST_HOOKS and a limit of 65536 polls (some ten milliseconds).  Every index stays in bounds; each call returns, its
// status says what happened, and the same call on the same workspace is right again once the hook is off.
#include <cstdio>
#include <cstring>
#include <vector>

#include "thrust_b200/merge.cuh"
#include "thrust_b200/reduce_by_key.cuh"
#include "thrust_b200/scan.cuh"
#include "thrust_b200/select.cuh"

static int failures = 0;
#define CHECK(cond) do { if (!(cond)) { std::printf("FAILED line %d: %s\n", __LINE__, #cond); ++failures; } } while (0)

constexpr size_t N = ((size_t)1 << 21) + 4099;
static int *d_in, *d_keys, *d_out, *d_out2, *d_merged;
static void* d_ws;
static std::vector<int> h_in, h_keys;

static unsigned status() {
  tb200::ws_header h;
  CHECK(cudaDeviceSynchronize() == cudaSuccess);
  CHECK(cudaMemcpy(&h, d_ws, sizeof(h), cudaMemcpyDeviceToHost) == cudaSuccess);
  return h.error;
}
static std::vector<int> back(const int* d, size_t n) { std::vector<int> h(n); CHECK(cudaMemcpy(h.data(), d, 4 * n, cudaMemcpyDeviceToHost) == cudaSuccess); return h; }

template <class Call, class Right> static void run_out(unsigned hook, Call call, Right right) {
  tb200::test_hook_flags() = hook;
  CHECK(call() == cudaSuccess);
  CHECK(status() == tb200::ERR_LOOKBACK_TIMEOUT);
  tb200::test_hook_flags() = 0;
  CHECK(call() == cudaSuccess);
  CHECK(status() == 0);
  right();
}

int main() {
  h_in.resize(N); h_keys.resize(N);
  for (size_t i = 0; i < N; ++i) { h_in[i] = (int)(i * 2654435761u % 1000); h_keys[i] = (int)(i / 5); }
  for (int** p : {&d_in, &d_keys, &d_out, &d_out2}) CHECK(cudaMalloc(p, 4 * N) == cudaSuccess);
  CHECK(cudaMalloc(&d_merged, 8 * N) == cudaSuccess && cudaMalloc(&d_ws, 64 << 20) == cudaSuccess);
  CHECK(cudaMemcpy(d_in, h_in.data(), 4 * N, cudaMemcpyHostToDevice) == cudaSuccess && cudaMemcpy(d_keys, h_keys.data(), 4 * N, cudaMemcpyHostToDevice) == cudaSuccess);
  std::vector<int> sums(N), kept, dropped;
  { int s = 0; for (size_t i = 0; i < N; ++i) sums[i] = s += h_in[i]; }
  const tb200::pred_lt pred{500};
  for (int x : h_in) (x < 500 ? kept : dropped).push_back(x);

  auto scan = [&] { return tb200::scan_async<true>((const int*)d_in, d_out, N, 0, false, tb200::plus_op(), d_ws, 0); };
  auto scanned = [&] { CHECK(back(d_out, N) == sums); };
  run_out(1, scan, scanned);
  run_out(1, [&] { return tb200::select_async<tb200::SEL_PRED, false>((const int*)d_in, (const int*)nullptr, d_out, (int*)nullptr, N, 0, pred, false, nullptr, d_ws, 0); },
          [&] { CHECK(back(d_out, kept.size()) == kept); });
  run_out(1, [&] { cudaMemcpyAsync(d_out, d_in, 4 * N, cudaMemcpyDeviceToDevice); return tb200::partition_inplace_async(d_out, d_out2, N, pred, nullptr, d_ws, 0); },
          [&] { std::vector<int> want(kept); want.insert(want.end(), dropped.begin(), dropped.end()); CHECK(back(d_out, N) == want); });
  run_out(1, [&] { return tb200::reduce_by_key_async((const int*)d_keys, (const int*)d_in, d_out, d_out2, N, 0, 0, tb200::equal_op(), tb200::plus_op(), nullptr, d_ws, 0); },
          [&] { std::vector<int> want((N + 4) / 5, 0); for (size_t i = 0; i < N; ++i) want[i / 5] += h_in[i]; CHECK(back(d_out2, want.size()) == want); });
  run_out(2, [&] { return tb200::merge_async<int, int, false>((const int*)d_keys, N, (const int*)d_keys, N, (const int*)nullptr, (const int*)nullptr, d_merged, (int*)nullptr,
                                                               tb200::less_op(), d_ws, 0); },
          [&] { std::vector<int> want(2 * N);
                for (size_t i = 0; i < 2 * N; ++i) want[i] = (int)(i / 10 < (N - 1) / 5 ? i / 10 : (N - 1) / 5); CHECK(back(d_merged, 2 * N) == want); });

  // a refused launch: the single-pass kernel serves the call
  CHECK(cudaMemset(d_out, 0, 4 * N) == cudaSuccess);
  tb200::test_hook_flags() = 4;
  CHECK(scan() == cudaSuccess);
  CHECK(status() == 0 && cudaGetLastError() == cudaSuccess);
  scanned();
  tb200::test_hook_flags() = 0;
  std::printf(failures ? "bounded_waits_test: %d FAILURES\n" : "bounded_waits_test: all checks passed\n", failures);
  return failures ? 1 : 0;
}
