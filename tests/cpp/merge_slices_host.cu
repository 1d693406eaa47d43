// Host check of how a tile's slices are cut out of two ranges (include/thrust_b200/merge.cuh), no GPU: every tile that
// is merged has its slices inside A and B and as many items as outputs, also where float keys hold NaNs and the
// comparator is no order on them.  Prints how many tiles were refused, with and without NaNs.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "thrust_b200/merge.cuh"

constexpr int TILE = 64;

static unsigned long long mix(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; z = (z ^ (z >> 27)) * 0x94D049BB133111EBull; return z ^ (z >> 31);
}

// returns the number of refused tiles, -1 if a tile that would be merged reaches outside
static int check(size_t na, size_t nb, int nan_per_mille, unsigned long long seed) {
  std::vector<float> a(na), b(nb);
  for (size_t i = 0; i < na; ++i) a[i] = (float)(mix(seed + i) % 100000);
  for (size_t i = 0; i < nb; ++i) b[i] = (float)(mix(seed + na + i) % 100000);
  std::sort(a.begin(), a.end()); std::sort(b.begin(), b.end());
  for (size_t i = 0; i < na; ++i) if ((int)(mix(seed + 77 + i) % 1000) < nan_per_mille) a[i] = NAN;
  for (size_t i = 0; i < nb; ++i) if ((int)(mix(seed + 99 + i) % 1000) < nan_per_mille) b[i] = NAN;
  tb200::merge_geometry g = tb200::merge_geometry::single(na, nb);
  g.cut(TILE);
  int refused = 0;
  for (size_t t = 0; t < g.num_tiles(); ++t) {
    size_t a0, alen, b0, blen, pair_out, local;
    g.locate<TILE>(t, a0, alen, b0, blen, pair_out, local);
    const size_t total = alen + blen;
    const unsigned tile_n = total - local < TILE ? (unsigned)(total - local) : (unsigned)TILE;
    auto split = [&](size_t diag) { return a0 + tb200::merge_path(a.data() + a0, alen, b.data() + b0, blen, diag, tb200::less_op()); };
    const tb200::merge_slices s(split(local), split(local + tile_n), a0, b0, local, tile_n);
    if (!s.consistent) { ++refused; continue; }
    if (s.na + s.nb != tile_n || s.a_begin + s.na > a0 + alen || s.b_begin + s.nb > b0 + blen || s.b_begin < b0) return -1;
  }
  return refused;
}

int main() {
  int plain = 0, with_nan = 0;
  for (int per_mille : {0, 2, 20, 100}) {
    for (int q = 0; q < 8; ++q) {
      const int r = check(20000 + 37 * q, q == 7 ? 3 : 30000 - 11 * q, per_mille, 1000ull * q);
      if (r < 0) { std::printf("a merged tile reaches outside its inputs\n"); return 1; }
      (per_mille ? with_nan : plain) += r;
    }
  }
  std::printf("refused: %d without NaNs, %d with\n", plain, with_nan);
  return plain == 0 && with_nan > 0 ? 0 : 1;
}
