// Host check (no GPU): the workspace that each algorithm asks for holds the descriptors of every route it may take, at
// sizes around whole tiles and with the single-pass kernels' tunables as given on the command line.
#include <cstdio>

#include "thrust_b200/reduce_by_key.cuh"
#include "thrust_b200/scan.cuh"
#include "thrust_b200/select.cuh"

using namespace tb200;
static int failures = 0;
static void check(const char* what, size_t n, size_t has, size_t needs) {
  if (has < sizeof(ws_header) + needs) { std::printf("%s, n = %zu: %zu bytes asked for, %zu used\n", what, n, has, sizeof(ws_header) + needs); ++failures; }
}
static size_t tiles_of(size_t n, size_t items) { return (n + items - 1) / items; }

template <class T> static void one_type(size_t n) {
  const size_t tiles = tiles_of(n, PIPE_TILE_BYTES / sizeof(T));
  check("scan plus", n, scan_workspace_bytes<T>(n), tile_chain<T, plus_op>::bytes(tiles));
  check("scan min", n, scan_workspace_bytes<T>(n), tile_chain<T, min_op>::bytes(tiles));
  check("select", n, select_workspace_bytes<T>(n), tile_chain<unsigned long long, plus_op>::bytes(tiles));
}
template <class K, class V> static void pair(size_t n) {
  check("reduce_by_key", n, rbk_workspace_bytes<K, V>(n), rbk_chain<V, plus_op>::bytes(tiles_of(n, rbk_pipe_shape<K, V>::ITEMS)));
}

int main() {
  for (size_t n : {(size_t)1 << 17, ((size_t)1 << 20) - 1, ((size_t)1 << 20) + 1, ((size_t)1 << 24) + 4099, (size_t)1 << 28, ((size_t)1 << 31) + 7}) {
    one_type<int>(n); one_type<unsigned>(n); one_type<float>(n); one_type<long long>(n); one_type<double>(n);
    pair<int, int>(n); pair<int, float>(n); pair<int, double>(n); pair<long long, float>(n); pair<long long, double>(n); pair<float, long long>(n);
  }
  return failures ? 1 : 0;
}
