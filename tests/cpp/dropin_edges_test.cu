// Corners of the drop-in, compiled like dropin_test.cu: in-place partition of plain arrays and of other iterators at ragged
// sizes, functors that must only ever see the caller's own elements, comparator sorts of keys around the size at which the
// sort's tile changes.  With THRUST_B200_LOG=1 in the environment the launches name the kernels that served the calls.
#include <thrust/device_vector.h>
#include <thrust/execution_policy.h>
#include <thrust/functional.h>
#include <thrust/host_vector.h>
#include <thrust/iterator/zip_iterator.h>
#include <thrust/merge.h>
#include <thrust/partition.h>
#include <thrust/reduce.h>
#include <thrust/sequence.h>
#include <thrust/sort.h>
#include <thrust/system_error.h>
#include <thrust/tuple.h>
#include <thrust/unique.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#ifndef THRUST_B200_OVERLAY_EXPECTED
#error "compile with -include thrust_b200/thrust_overlay.cuh -DTHRUST_B200_OVERLAY_EXPECTED"
#endif

static int failures = 0;
#define CHECK(cond) do { if (!(cond)) { std::printf("FAILED line %d: %s\n", __LINE__, #cond); ++failures; } } while (0)

static unsigned long long mix(unsigned long long i) {
  unsigned long long z = i + 0x9E3779B97F4A7C15ull * 7;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; z = (z ^ (z >> 27)) * 0x94D049BB133111EBull; return z ^ (z >> 31);
}

// ---- in-place partition
template <class T> struct below { T bound; __host__ __device__ bool operator()(const T& x) const { return x < bound; } };
template <class T> static void check_partition(int n) {
  std::vector<T> h(n);
  for (int i = 0; i < n; ++i) h[i] = (T)(mix(i) % 1000);
  for (int bound : {0, 500, 1000}) {
    thrust::device_vector<T> d(h.begin(), h.end());
    std::vector<T> want(h);
    const auto wmid = std::stable_partition(want.begin(), want.end(), below<T>{(T)bound});
    const auto mid = thrust::stable_partition(thrust::device, d.begin(), d.end(), below<T>{(T)bound});
    thrust::host_vector<T> got = d;
    CHECK(mid - d.begin() == wmid - want.begin() && std::equal(want.begin(), want.end(), got.begin()));
    d = h;   // one item into the vector: off a 16-byte boundary
    const auto mid1 = thrust::partition(thrust::device, d.begin() + 1, d.end(), below<T>{(T)bound});
    CHECK(mid1 - (d.begin() + 1) == std::count_if(h.begin() + 1, h.end(), below<T>{(T)bound}));
    CHECK((thrust::is_partitioned(thrust::device, d.begin() + 1, d.end(), below<T>{(T)bound})));
  }
}
struct first_below { int bound; template <class Z> __host__ __device__ bool operator()(const Z& z) const { return thrust::get<0>(z) < bound; } };

// ---- functors that report an argument which is not one of the caller's elements
struct same_in_range {
  int lo, hi; int* strange;
  __device__ bool operator()(int a, int b) const { if (a < lo || a > hi || b < lo || b > hi) atomicExch(strange, 1); return a == b; }
};
static void check_functors(int n) {
  std::vector<int> h(n);
  for (int i = 0; i < n; ++i) h[i] = 1000000 + i / 3;
  const int runs = (n + 2) / 3;
  thrust::device_vector<int> d(h.begin(), h.end()), out(n), ones(n, 1), sums(n), strange(1, 0);
  const same_in_range eq{1000000, h.back(), thrust::raw_pointer_cast(strange.data())};
  // leave other numbers in shared memory first: a reduction over small values
  thrust::device_vector<int> noise(1 << 22, 7);
  thrust::sort(thrust::device, noise.begin(), noise.end());
  CHECK(thrust::unique_copy(thrust::device, d.begin(), d.end(), out.begin(), eq) - out.begin() == runs);
  CHECK(strange[0] == 0);
  const auto e = thrust::reduce_by_key(thrust::device, d.begin(), d.end(), ones.begin(), out.begin(), sums.begin(), eq);
  CHECK(e.first - out.begin() == runs && thrust::reduce(thrust::device, sums.begin(), e.second, 0) == n);
  CHECK(strange[0] == 0);
}

// ---- what the kernels report comes out as the exception's text
static void check_report(int n) {
  std::vector<float> a(n), b(n);
  for (int i = 0; i < n; ++i) { a[i] = (float)i; b[i] = (float)i; if (mix(i) % 10 == 0) a[i] = NAN; if (mix(i + n) % 10 == 0) b[i] = NAN; }
  thrust::device_vector<float> da(a.begin(), a.end()), db(b.begin(), b.end()), dm(2 * n);
  try { thrust::merge(thrust::device, da.begin(), da.end(), db.begin(), db.end(), dm.begin()); }
  catch (const thrust::system_error& e) { CHECK(std::strstr(e.what(), "two looks at a tile disagree") != nullptr); return; }
  CHECK(!"a merge of ranges that are not sorted went unnoticed");
}

// ---- comparator sorts of struct keys
template <int WORDS> struct key { int w[WORDS]; };
struct by_first_word { template <class K> __host__ __device__ bool operator()(const K& a, const K& b) const { return a.w[0] < b.w[0]; } };
template <int WORDS> static void check_sort(int n) {
  std::vector<key<WORDS>> h(n);
  for (int i = 0; i < n; ++i) for (int q = 0; q < WORDS; ++q) h[i].w[q] = q == 0 ? (int)(mix(i) % 5000) : i * WORDS + q;
  thrust::device_vector<key<WORDS>> d(h.begin(), h.end());
  thrust::stable_sort(thrust::device, d.begin(), d.end(), by_first_word());
  std::stable_sort(h.begin(), h.end(), by_first_word());
  thrust::host_vector<key<WORDS>> got = d;
  bool ok = true;
  for (int i = 0; i < n && ok; ++i) for (int q = 0; q < WORDS; ++q) ok = ok && got[i].w[q] == h[i].w[q];
  CHECK(ok);
}

int main() {
  for (int n : {1, 1000, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, 1500007}) { check_partition<int>(n); check_partition<double>(n); }
  check_partition<short>(300001);
  check_partition<float>((1 << 24) + 4099);
  { const int n = 300007; thrust::device_vector<int> a(n), b(n); thrust::sequence(a.begin(), a.end()); thrust::sequence(b.begin(), b.end());
    const auto z = thrust::make_zip_iterator(thrust::make_tuple(a.begin(), b.begin()));
    CHECK(thrust::stable_partition(thrust::device, z, z + n, first_below{1000}) - z == 1000); }
  check_functors(1 << 18);
  check_functors(3000001);
  check_report(200003);
  check_sort<4>(50021); check_sort<5>(50021); check_sort<5>(100); check_sort<6>(50021);
  if (cudaDeviceSynchronize() != cudaSuccess) { std::printf("FAILED: sticky CUDA error\n"); ++failures; }
  std::printf(failures ? "dropin_edges_test: %d FAILURES\n" : "dropin_edges_test: all checks passed\n", failures);
  return failures ? 1 : 0;
}
