// Merge-path merge and merge sort for sm_100a.
//
// merge / merge_by_key (replaces PartitionAgent + MergeAgent of
// thrust/system/cuda/detail/merge.h:152-660): a first kernel finds, for every output tile boundary, how
// many items of range A precede it (search along the merge-path diagonal); then every thread of a tile
// finds its own start with a second merge-path search in shared memory and merges its outputs serially.
// Ties take from A first, so the merge is stable.  Two kernels do that:
//   merge_slices_kernel   plain arrays of 4- and 8-byte keys and payloads: bulk copies bring the tile's slices,
//                         the merge records source positions, keys and payloads are gathered by them;
//   merge_kernel          any iterators and sizes: loads and results pass through shared memory.
//
// merge sort (replaces BlockSortAgent + PartitionAgent + MergeAgent of
// thrust/system/cuda/detail/sort.h:235-1138): block_sort_kernel sorts each tile (per-thread
// odd-even transposition network, then log2(BLOCK) rounds of pairwise merge-path merges in
// shared memory, all stable), and the same merge kernels run in "pairwise" mode over runs of
// doubling length, ping-ponging between the data and a scratch copy.
#pragma once
#include "bulk_copy.cuh"
#include "common.cuh"

namespace tb200 {

constexpr int MERGE_BLOCK = 256;
// Tunables of merge_kernel: items per thread and resident CTAs per SM asked of the compiler (a register cap)
// for items of up to 8 and up to 12 bytes (key + payload).  It is bound by the latency of its
// barrier-separated phases and by the shared-memory pipe, so small tiles and many resident CTAs pay:
// 15 / 11 items at the compiler's own 58 registers (4 CTAs per SM) took 1.2 to 1.7 times as long.
#ifndef TB200_MERGE_IPT8
#define TB200_MERGE_IPT8 11
#endif
#ifndef TB200_MERGE_IPT12
#define TB200_MERGE_IPT12 7
#endif
#ifndef TB200_MERGE_CTAS8
#define TB200_MERGE_CTAS8 8
#endif
#ifndef TB200_MERGE_CTAS12
#define TB200_MERGE_CTAS12 7
#endif
#ifndef TB200_BSORT_IPT8
#define TB200_BSORT_IPT8 16
#endif
#ifndef TB200_BSORT_CTAS8
#define TB200_BSORT_CTAS8 5
#endif

// Items per thread: tuned for the small types, then whatever keeps the staged tile (keys and
// payloads of 256 * IPT items) inside 44 KB of static shared memory, as the reference sizes its
// tiles by sizeof(T) (thrust/system/cuda/detail/merge.h:301-360).
constexpr int MERGE_SMEM_BUDGET = 44 * 1024;
template <int KB, int VB> struct merge_tuning {
  static constexpr int TUNED = (KB + VB) <= 8 ? TB200_MERGE_IPT8 : ((KB + VB) <= 12 ? TB200_MERGE_IPT12 : 9);
  static constexpr int MIN_CTAS = (KB + VB) <= 8 ? TB200_MERGE_CTAS8 : ((KB + VB) <= 12 ? TB200_MERGE_CTAS12 : 1);
  static constexpr int FIT = MERGE_SMEM_BUDGET / (MERGE_BLOCK * (KB + VB));
  static constexpr int IPT = TUNED < FIT ? TUNED : (FIT < 1 ? 1 : FIT);
  static_assert(MERGE_BLOCK * IPT * (KB + VB) + KB <= 48 * 1024, "key + payload too large for the merge tile (more than 160 bytes per item)");
};

// Number of items taken from A among the first `diag` outputs of merge(A[0,na), B[0,nb)).
template <class KeyItA, class KeyItB, class Comp>
__host__ __device__ __forceinline__ size_t merge_path(KeyItA a, size_t na, KeyItB b, size_t nb, size_t diag, Comp comp) {
  size_t lo = diag > nb ? diag - nb : 0;
  size_t hi = diag < na ? diag : na;
  while (lo < hi) {
    size_t mid = (lo + hi) >> 1;
    if (!comp(b[diag - 1 - mid], a[mid])) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Which slices a tile merges.  The output is cut into "pairs": in single mode one pair, A = [0, na)
// of one array and B = [0, nb) of another; in pairwise mode (merge sort) one array of n items in
// sorted runs of length `run`, pair p merging runs 2p and 2p+1.  Tiles never straddle a pair:
// each pair is covered by tiles_per_pair tiles of TILE outputs (cut() sets it).
struct merge_geometry {
  size_t na, nb;          // single mode
  size_t n, run;          // pairwise mode (run == 0 selects single mode)
  size_t tiles_per_pair;
  static merge_geometry single(size_t na, size_t nb) { merge_geometry g; g.na = na; g.nb = nb; g.n = na + nb; g.run = 0; g.tiles_per_pair = 1; return g; }
  static merge_geometry pairwise(size_t n, size_t run) { merge_geometry g; g.na = g.nb = 0; g.n = n; g.run = run; g.tiles_per_pair = 1; return g; }
  void cut(size_t tile) { tiles_per_pair = ((run == 0 ? na + nb : 2 * run) + tile - 1) / tile; if (tiles_per_pair == 0) tiles_per_pair = 1; }
  __host__ __device__ size_t num_tiles() const {
    if (run == 0) return tiles_per_pair;
    return (n + 2 * run - 1) / (2 * run) * tiles_per_pair;
  }
  // tile t -> its pair's slices (offsets into the A / B arrays), the pair's first output position
  // and the tile's first output position relative to that
  template <int TILE>
  __host__ __device__ void locate(size_t t, size_t& a0, size_t& alen, size_t& b0, size_t& blen, size_t& pair_out, size_t& local) const {
    const size_t p = t / tiles_per_pair;
    local = (t % tiles_per_pair) * (size_t)TILE;
    if (run == 0) { a0 = 0; alen = na; b0 = 0; blen = nb; pair_out = 0; return; }
    pair_out = p * 2 * run;
    a0 = pair_out;
    alen = n - a0 < run ? n - a0 : run;
    b0 = a0 + alen;
    blen = n - b0 < run ? n - b0 : run;
  }
};

// A tile's slices of A and B, from the splits of its two diagonals.  Each split lies inside its own diagonal's bounds
// whatever the comparator answers; under one that is no strict weak order on the data (keys that are NaN) two
// neighbouring splits need not agree, and then the slices are no ranges: `consistent` is false and the tile must not be merged.
struct merge_slices {
  size_t a_begin, b_begin;
  unsigned na, nb;
  bool consistent;
  __host__ __device__ merge_slices(size_t split_begin, size_t split_end, size_t a0, size_t b0, size_t local, unsigned tile_n)
      : a_begin(split_begin), b_begin(b0 + local - (split_begin - a0)), na((unsigned)(split_end - split_begin)), nb(tile_n - na),
        consistent(split_end >= split_begin && split_end - split_begin <= tile_n) {}
};

// One thread per tile: where in A the tile's outputs start and end.
template <class KeyItA, class KeyItB, class Comp, int TILE>
__global__ void __launch_bounds__(256)
merge_partition_kernel(KeyItA ka, KeyItB kb, merge_geometry g, size_t num_tiles, Comp comp, size_t* a_split) {
  size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= num_tiles) return;
  size_t a0, alen, b0, blen, pair_out, local;
  g.locate<TILE>(t, a0, alen, b0, blen, pair_out, local);
  const size_t pair_total = alen + blen;
  size_t d0 = local < pair_total ? local : pair_total;
  size_t d1 = local + TILE < pair_total ? local + TILE : pair_total;
  a_split[2 * t] = a0 + merge_path(ka + a0, alen, kb + b0, blen, d0, comp);
  a_split[2 * t + 1] = a0 + merge_path(ka + a0, alen, kb + b0, blen, d1, comp);
}

template <class KeyItA, class KeyItB, class ValItA, class ValItB, class KeyOutIt, class ValOutIt, class K, class V, bool HAS_V, class Comp, int IPT>
__global__ void __launch_bounds__(MERGE_BLOCK, merge_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>::MIN_CTAS)
merge_kernel(KeyItA ka, KeyItB kb, ValItA va, ValItB vb, KeyOutIt ko, ValOutIt vo, merge_geometry g, Comp comp, const size_t* a_split, unsigned* err) {
  constexpr int TILE = MERGE_BLOCK * IPT;
  TB200_SHARED_ARRAY(K, s_key, TILE + 1);
  TB200_SHARED_ARRAY(V, s_val, HAS_V ? TILE : 1);
  const size_t t = blockIdx.x;
  size_t a0p, alen, b0p, blen, pair_out, local;
  g.locate<TILE>(t, a0p, alen, b0p, blen, pair_out, local);
  const size_t pair_total = alen + blen;
  if (local >= pair_total) return;                       // a short last pair leaves its later tiles empty
  const size_t out0 = pair_out + local;
  const unsigned tile_n = pair_total - local < TILE ? (unsigned)(pair_total - local) : (unsigned)TILE;
  const merge_slices slices(a_split[2 * t], a_split[2 * t + 1], a0p, b0p, local, tile_n);
  if (!slices.consistent) { if (threadIdx.x == 0) record_error(err, ERR_INCONSISTENT); return; }
  const size_t a_begin = slices.a_begin, b_begin = slices.b_begin;
  const unsigned na = slices.na, nb = slices.nb;

  // ---- stage both key slices: A at [0, na), B at [na, na + nb)
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    unsigned c = threadIdx.x + i * MERGE_BLOCK;
    if (c < tile_n) stash(&s_key[c], c < na ? (K)ka[a_begin + c] : (K)kb[b_begin + (c - na)]);
  }
  __syncthreads();

  // ---- per-thread merge path + serial merge of IPT outputs
  unsigned d0 = threadIdx.x * IPT; if (d0 > tile_n) d0 = tile_n;
  unsigned ai = (unsigned)merge_path(s_key, (size_t)na, s_key + na, (size_t)nb, (size_t)d0, comp);
  unsigned bi = d0 - ai;
  K out_k[IPT]; unsigned short src[IPT];
  K keyA = ai < na ? s_key[ai] : K();
  K keyB = bi < nb ? s_key[na + bi] : K();
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    bool take_b = (bi < nb) && (ai >= na || comp(keyB, keyA));
    out_k[i] = take_b ? keyB : keyA;
    src[i] = (unsigned short)(take_b ? na + bi : ai);
    if (take_b) { ++bi; keyB = bi < nb ? s_key[na + bi] : keyB; }
    else { ++ai; keyA = ai < na ? s_key[ai] : keyA; }
  }
  __syncthreads();
  // ---- keys out through shared memory (thread's outputs are consecutive; stores become coalesced)
#pragma unroll
  for (int i = 0; i < IPT; ++i) { unsigned j = threadIdx.x * IPT + i; if (j < tile_n) stash(&s_key[j], out_k[i]); }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < IPT; ++i) { unsigned c = threadIdx.x + i * MERGE_BLOCK; if (c < tile_n) ko[out0 + c] = s_key[c]; }

  if constexpr (HAS_V) {
    V v_in[IPT];
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      unsigned c = threadIdx.x + i * MERGE_BLOCK;
      if (c < tile_n) v_in[i] = c < na ? (V)va[a_begin + c] : (V)vb[b_begin + (c - na)];
    }
#pragma unroll
    for (int i = 0; i < IPT; ++i) { unsigned c = threadIdx.x + i * MERGE_BLOCK; if (c < tile_n) stash(&s_val[c], v_in[i]); }
    __syncthreads();
    V out_v[IPT];
#pragma unroll
    for (int i = 0; i < IPT; ++i) { unsigned j = threadIdx.x * IPT + i; if (j < tile_n) out_v[i] = s_val[src[i]]; }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < IPT; ++i) { unsigned j = threadIdx.x * IPT + i; if (j < tile_n) stash(&s_val[j], out_v[i]); }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < IPT; ++i) { unsigned c = threadIdx.x + i * MERGE_BLOCK; if (c < tile_n) vo[out0 + c] = s_val[c]; }
  }
}

// ---------------------------------------------------------------- merge of contiguous arrays
// The kernel for plain arrays of 4- and 8-byte keys and payloads.  merge_kernel above is bound by the
// shared-memory pipe: staging stores, the keys' way back through shared memory, three accesses per payload.
// Here the copy engine brings the four slices (keys and payloads of A and B) into shared memory, the merge
// leaves only each output's source position there (16 bits; a thread's eight in one 16-byte store), and
// keys and payloads are gathered by it straight into the coalesced stores: two barriers instead of eight and
// about half the shared-memory wavefronts.  Measured on B200 against merge_kernel: 2 x 2^27 (u64, u32) 1.46 ms
// (1.73), (u32, u32) 0.97 ms (1.31), 2 x 4 M (u64, u32) 57 us (84), 2 x 50 k 16 us (22).
template <int KB, int VB> struct merge_slices_tuning {
  static constexpr int IPT = 8;                          // source positions of a thread: one 16-byte store
  static constexpr int TILE = MERGE_BLOCK * IPT;
  // a slice keeps its distance from a 16-byte boundary, so up to 15 bytes are lost in front of A, behind it and in front of B;
  // the merge's reads end one item behind the last of TILE at most
  static constexpr int KEY_BYTES = TILE * KB + 48, VAL_BYTES = VB ? TILE * VB + 48 : 0;
  static constexpr int MIN_CTAS = KB + VB <= 8 ? 8 : KB + VB <= 12 ? 7 : 6;   // as many as shared memory holds
};

// Items [0, n) at `src` to the same offsets of `dst`, which has src's distance from a 16-byte boundary: the
// 16-byte pieces inside by one bulk copy (thread `issuer`; returns its bytes to every caller), the ragged ends
// by the lanes of one warp.
template <class T> __device__ __forceinline__ unsigned slice_head(const T* src, unsigned n) {
  const unsigned h = (unsigned)((16 - (reinterpret_cast<uintptr_t>(src) & 15)) & 15) / sizeof(T);
  return h < n ? h : n;
}
template <class T> __device__ __forceinline__ unsigned slice_bulk_bytes(const T* src, unsigned n) {
  return (unsigned)((n - slice_head(src, n)) * sizeof(T)) & ~15u;
}
template <class T> __device__ __forceinline__ void slice_issue(T* dst, const T* src, unsigned n, unsigned long long* bar, unsigned long long policy) {
  const unsigned bytes = slice_bulk_bytes(src, n), h = slice_head(src, n);
  if (bytes) bulk_load(dst + h, src + h, bytes, bar, policy);
}
template <class T> __device__ __forceinline__ void slice_ends(T* dst, const T* src, unsigned n) {
  const unsigned h = slice_head(src, n), t = h + slice_bulk_bytes(src, n) / sizeof(T), lane = lane_id();
  if (lane < h) dst[lane] = src[lane];
  if (t + lane < n) dst[t + lane] = src[t + lane];   // fewer than 16 / sizeof(T) items
}

// Where diagonal `diag` of merge(a[0, alen), b[0, blen)) is split, by a warp with 32 probes per round trip, so that the search over
// 2^k items takes k / 5 of them instead of k.  The same result in every lane.
template <class K, class Comp>
__device__ __forceinline__ size_t warp_merge_path(const K* a, size_t alen, const K* b, size_t blen, size_t diag, Comp comp) {
  size_t lo = diag > blen ? diag - blen : 0, hi = diag < alen ? diag : alen;
  while (lo < hi) {
    const size_t step = (hi - lo + 31) / 32, mid = lo + lane_id() * step;
    const unsigned below = __popc(__ballot_sync(FULL_MASK, mid < hi && !comp(b[diag - 1 - mid], a[mid])));   // a prefix of the lanes
    if (below < 32 && lo + below * step < hi) hi = lo + below * step;
    if (below) lo += (below - 1) * step + 1;
  }
  return lo;
}

// First item of A in every tile, by a warp per tile: few round trips, which is what a small input waits for.
template <class K, class Comp, int TILE>
__global__ void __launch_bounds__(256)
merge_split_kernel(const K* ka, const K* kb, merge_geometry g, unsigned num_tiles, Comp comp, size_t* a_split) {
  grid_dependents_launch();
  grid_dependency_wait();
  const unsigned t = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (t >= num_tiles) return;
  size_t a0, alen, b0, blen, pair_out, local;
  g.locate<TILE>(t, a0, alen, b0, blen, pair_out, local);
  const size_t total = alen + blen;
  const size_t lo = warp_merge_path(ka + a0, alen, kb + b0, blen, local < total ? local : total, comp);
  if (lane_id() == 0) a_split[t] = a0 + lo;
}

// The same for many tiles, a thread per tile.  What bounds it there is the number of scattered 32-byte reads: a warp per tile
// makes 64 of them in each round trip that misses.  Here two warps find the splits of the CTA's first and last diagonal,
// which bound all splits between; a thread starts from where the split would lie if A and B were evenly mixed
// in between, widens its step until the split is passed, and halves.
constexpr int SPLIT_GROUP = 256;   // tiles of a CTA
template <class K, class Comp, int TILE>
__global__ void __launch_bounds__(SPLIT_GROUP)
merge_split_group_kernel(const K* ka, const K* kb, merge_geometry g, unsigned groups_per_pair, Comp comp, size_t* a_split) {
  __shared__ size_t s_end[2];
  grid_dependents_launch();
  grid_dependency_wait();
  const size_t pair = blockIdx.x / groups_per_pair, first = (size_t)(blockIdx.x % groups_per_pair) * SPLIT_GROUP;   // inside the pair
  const size_t in_pair = first + threadIdx.x, t = pair * g.tiles_per_pair + in_pair;
  size_t a0, alen, b0, blen, pair_out, local;
  g.locate<TILE>(pair * g.tiles_per_pair, a0, alen, b0, blen, pair_out, local);
  const size_t total = alen + blen;
  const K* a = ka + a0;
  const K* b = kb + b0;
  auto diag_of = [&](size_t tile) { const size_t d = tile * TILE; return d < total ? d : total; };
  const size_t d0 = diag_of(first), d1 = diag_of(first + SPLIT_GROUP);
  const int warp = threadIdx.x >> 5;
  if (warp < 2) {
    const size_t s = warp_merge_path(a, alen, b, blen, warp ? d1 : d0, comp);
    if (lane_id() == 0) s_end[warp] = s;
  }
  __syncthreads();
  if (in_pair >= g.tiles_per_pair) return;
  const size_t diag = diag_of(in_pair), s0 = s_end[0], s1 = s_end[1];
  size_t lo = diag > blen ? diag - blen : 0, hi = diag < alen ? diag : alen;
  // a split lies between those of earlier and later diagonals (under a comparator that is no order it need not; then the
  // diagonal's own bounds stand, as everywhere)
  const size_t lo2 = lo > s0 ? lo : s0, hi2 = hi < s1 ? hi : s1;
  if (lo2 <= hi2) { lo = lo2; hi = hi2; }
  auto past = [&](size_t mid) { return !comp(b[diag - 1 - mid], a[mid]); };   // the split lies behind item `mid`
  if (lo < hi) {
    size_t mid = s1 > s0 && d1 > d0 ? s0 + (size_t)((double)(s1 - s0) * (double)(diag - d0) / (double)(d1 - d0)) : lo;
    mid = mid < lo ? lo : mid >= hi ? hi - 1 : mid;
    size_t width = 64;
    if (past(mid)) {
      lo = mid + 1;
      while (lo < hi) {
        mid = hi - lo > width ? lo + width : hi - 1;
        if (past(mid)) { lo = mid + 1; width *= 4; } else { hi = mid; break; }
      }
    } else {
      hi = mid;
      while (lo < hi) {
        mid = hi - lo > width ? hi - width : lo;
        if (past(mid)) { lo = mid + 1; break; } else { hi = mid; width *= 4; }
      }
    }
    while (lo < hi) {
      mid = (lo + hi) >> 1;
      if (past(mid)) lo = mid + 1; else hi = mid;
    }
  }
  a_split[t] = a0 + lo;
}

template <class K, class V, bool HAS_V, class Comp>
__global__ void __launch_bounds__(MERGE_BLOCK, (merge_slices_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>::MIN_CTAS))
merge_slices_kernel(const K* ka, const K* kb, const V* va, const V* vb, K* ko, V* vo, merge_geometry g, Comp comp, const size_t* a_split, unsigned* err) {
  using Tuning = merge_slices_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>;
  constexpr int IPT = Tuning::IPT, TILE = Tuning::TILE;
  __shared__ __align__(16) unsigned char s_keys[Tuning::KEY_BYTES];
  __shared__ __align__(16) unsigned char s_vals[HAS_V ? Tuning::VAL_BYTES : 16];
  __shared__ __align__(16) unsigned short s_src[TILE];
  __shared__ unsigned long long bars[2];               // the keys' slices have arrived, the payloads'
  __shared__ size_t s_split[2];
  grid_dependents_launch();
  grid_dependency_wait();
  const unsigned t = blockIdx.x;
  size_t a0p, alen, b0p, blen, pair_out, local;
  g.locate<TILE>(t, a0p, alen, b0p, blen, pair_out, local);
  const size_t pair_total = alen + blen;
  if (local >= pair_total) return;                     // a short last pair leaves its later tiles empty
  const unsigned tile_n = pair_total - local < TILE ? (unsigned)(pair_total - local) : (unsigned)TILE;
  const int warp = threadIdx.x >> 5;
  if (!a_split) {   // no pass before this one has found the splits: two warps do
    if (warp < 2) {
      const size_t s = a0p + warp_merge_path(ka + a0p, alen, kb + b0p, blen, warp ? local + tile_n : local, comp);
      if (lane_id() == 0) s_split[warp] = s;
    }
    __syncthreads();
  }
  const size_t split_begin = a_split ? a_split[t] : s_split[0];
  const size_t split_end = !a_split ? s_split[1] : local + TILE < pair_total ? a_split[t + 1] : a0p + alen;
  const merge_slices slices(split_begin, split_end, a0p, b0p, local, tile_n);
  if (!slices.consistent) { if (threadIdx.x == 0) record_error(err, ERR_INCONSISTENT); return; }   // before any copy is sized by them
  const size_t a_begin = slices.a_begin, b_begin = slices.b_begin;
  const unsigned na = slices.na, nb = slices.nb;
  auto phase = [](const void* p) { return (unsigned)(reinterpret_cast<uintptr_t>(p) & 15); };

  // ---- the slices' places: A first, B behind it on the next 16-byte boundary, each shifted by its phase
  const unsigned ka_at = phase(ka + a_begin), kb_at = ((ka_at + na * (unsigned)sizeof(K) + 15) & ~15u) + phase(kb + b_begin);
  K* const sk_a = reinterpret_cast<K*>(s_keys + ka_at);
  K* const sk_b = reinterpret_cast<K*>(s_keys + kb_at);
  V* sv_a = nullptr;
  V* sv_b = nullptr;
  if constexpr (HAS_V) {
    const unsigned va_at = phase(va + a_begin), vb_at = ((va_at + na * (unsigned)sizeof(V) + 15) & ~15u) + phase(vb + b_begin);
    sv_a = reinterpret_cast<V*>(s_vals + va_at);
    sv_b = reinterpret_cast<V*>(s_vals + vb_at);
  }
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 1);
    if (HAS_V) mbar_init(&bars[1], 1);
    mbar_init_fence();
    const unsigned long long policy = l2_stream_policy();
    unsigned awaited = slice_bulk_bytes(ka + a_begin, na) + slice_bulk_bytes(kb + b_begin, nb);
#ifdef TB200_TEST_HOOKS
    if (reinterpret_cast<const ws_header*>(err)->flags & 2u) awaited += 16;   // err points at the header's first word
#endif
    mbar_arrive_expect(&bars[0], awaited);
    slice_issue(sk_a, ka + a_begin, na, &bars[0], policy);
    slice_issue(sk_b, kb + b_begin, nb, &bars[0], policy);
    if constexpr (HAS_V) {
      mbar_arrive_expect(&bars[1], slice_bulk_bytes(va + a_begin, na) + slice_bulk_bytes(vb + b_begin, nb));
      slice_issue(sv_a, va + a_begin, na, &bars[1], policy);
      slice_issue(sv_b, vb + b_begin, nb, &bars[1], policy);
    }
  }
  if (warp == 1) slice_ends(sk_a, ka + a_begin, na);
  if (warp == 2) slice_ends(sk_b, kb + b_begin, nb);
  if constexpr (HAS_V) {
    if (warp == 3) slice_ends(sv_a, va + a_begin, na);
    if (warp == 4) slice_ends(sv_b, vb + b_begin, nb);
  }
  __syncthreads();
  // bounded: reported after the limit, given up after twice that (the CTA should not end while its copies are in flight)
  auto wait = [&](unsigned long long* bar) {
    for (unsigned iter = 0; !mbar_try_wait(bar, 0) && iter < 2 * MBAR_SPIN_LIMIT; ++iter)
      if (iter == MBAR_SPIN_LIMIT) record_error(err, ERR_LOOKBACK_TIMEOUT);
  };
  wait(&bars[0]);

  // ---- per-thread merge path, then a serial merge that records where each output comes from
  unsigned d0 = threadIdx.x * IPT; if (d0 > tile_n) d0 = tile_n;
  unsigned ai, bi;
  {
    unsigned lo = d0 > nb ? d0 - nb : 0, hi = d0 < na ? d0 : na;
    while (lo < hi) {
      const unsigned mid = (lo + hi) >> 1;
      if (!comp(sk_b[d0 - 1 - mid], sk_a[mid])) lo = mid + 1; else hi = mid;
    }
    ai = lo; bi = d0 - lo;
  }
  unsigned packed[IPT / 2];
  // the candidates stay in registers; only the side that was taken is read again, always: past a slice's end that is some
  // word inside s_keys which nothing looks at, and a load under no condition is cheaper than one under two (2 x 2^27
  // (u64, u32) 1.41 ms against 1.47)
  K key_a = sk_a[ai], key_b = sk_b[bi];
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const bool take_b = bi < nb && (ai >= na || comp(key_b, key_a));
    const unsigned src = take_b ? na + bi : ai;
    if (i & 1) packed[i / 2] |= src << 16; else packed[i / 2] = src;
    ai += take_b ? 0u : 1u;
    bi += take_b ? 1u : 0u;
    const K next = *(take_b ? sk_b + bi : sk_a + ai);
    key_b = take_b ? next : key_b;
    key_a = take_b ? key_a : next;
  }
  *reinterpret_cast<uint4*>(s_src + threadIdx.x * IPT) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  if constexpr (HAS_V) wait(&bars[1]);
  __syncthreads();

  // ---- consecutive threads on consecutive outputs
  const size_t out0 = pair_out + local;
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const unsigned c = threadIdx.x + i * MERGE_BLOCK;
    if (c < tile_n) {
      const unsigned src = s_src[c];
      const bool from_b = src >= na;
      ko[out0 + c] = from_b ? sk_b[src - na] : sk_a[src];
      if constexpr (HAS_V) vo[out0 + c] = from_b ? sv_b[src - na] : sv_a[src];
    }
  }
}

// Whether merge_slices_kernel may serve a call: plain arrays of the key and payload types.
template <class T> struct merge_slice_type { static constexpr bool value = std::is_trivially_copyable<T>::value && (sizeof(T) == 4 || sizeof(T) == 8) && alignof(T) == sizeof(T); };
template <class It, class T> struct is_array_of : std::false_type {};
template <class T> struct is_array_of<T*, T> : std::true_type {};
template <class T> struct is_array_of<const T*, T> : std::true_type {};
template <class K, class V, bool HAS_V, class KeyItA, class KeyItB, class ValItA, class ValItB, class KeyOutIt, class ValOutIt> struct merge_slices_ok {
  static constexpr bool keys = merge_slice_type<K>::value && is_array_of<KeyItA, K>::value && is_array_of<KeyItB, K>::value && is_array_of<KeyOutIt, K>::value;
  static constexpr bool vals = !HAS_V || (merge_slice_type<V>::value && is_array_of<ValItA, V>::value && is_array_of<ValItB, V>::value && is_array_of<ValOutIt, V>::value);
  static constexpr bool value = keys && vals;
};

template <class K, class V, bool HAS_V> constexpr int merge_tile_items() { return MERGE_BLOCK * merge_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>::IPT; }

template <class K, class V, bool HAS_V> size_t merge_workspace_bytes(size_t total) {
  // pairwise passes round every pair up to whole tiles: at most one extra tile per pair, and a pair
  // is never smaller than a block-sort tile, so 2x the single-mode tile count is a safe bound
  constexpr size_t slices = merge_slices_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>::TILE, items = merge_tile_items<K, V, HAS_V>();
  constexpr size_t tile = slices < items ? slices : items;   // either kernel may run
  size_t tiles = (total + tile - 1) / tile;
  return sizeof(ws_header) + align_up((4 * tiles + 8) * sizeof(size_t), 256);
}

// The splits of a pass.  Beyond 4096 tiles a thread per tile is faster on every shape tried (2 x 2^26 u64, microseconds here /
// a warp per tile: 39 / 201 uniform, 29 / 164 normal against uniform, 57 / 184 with 1000 distinct values, 12 / 164 disjoint;
// 16384 tiles in sorted runs of 2^12 20 / 25, of 2^17 16 / 37); at 4096 tiles both take 18, at 1024 it is 16 / 10.
constexpr unsigned SPLIT_WARP_TILES = 4096;
template <class K, class Comp, int TILE>
cudaError_t merge_split_async(const K* ka, const K* kb, const merge_geometry& g, unsigned tiles, Comp comp, size_t* a_split, bool overlap, cudaStream_t stream) {
  if (tiles <= SPLIT_WARP_TILES) return launch_after(merge_split_kernel<K, Comp, TILE>, (tiles + 7) / 8, 256, 0, stream, ka, kb, g, tiles, comp, a_split);
  const unsigned groups = (unsigned)((g.tiles_per_pair + SPLIT_GROUP - 1) / SPLIT_GROUP), grid = (unsigned)(tiles / g.tiles_per_pair) * groups;
  if (overlap) return launch_after(merge_split_group_kernel<K, Comp, TILE>, grid, SPLIT_GROUP, 0, stream, ka, kb, g, groups, comp, a_split);
  merge_split_group_kernel<K, Comp, TILE><<<grid, SPLIT_GROUP, 0, stream>>>(ka, kb, g, groups, comp, a_split);
  return cudaGetLastError();
}

// One merge pass (single or pairwise geometry); no sync.
template <class K, class V, bool HAS_V, class KeyItA, class KeyItB, class ValItA, class ValItB, class KeyOutIt, class ValOutIt, class Comp>
cudaError_t merge_pass_async(KeyItA ka, KeyItB kb, ValItA va, ValItB vb, KeyOutIt ko, ValOutIt vo, merge_geometry g, Comp comp, void* ws,
                             cudaStream_t stream) {
  constexpr int IPT = merge_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>::IPT;
  constexpr int TILE = MERGE_BLOCK * IPT;
  if (g.n == 0) return cudaSuccess;
  size_t* a_split = reinterpret_cast<size_t*>(static_cast<char*>(ws) + sizeof(ws_header));
  ws_header* const hdr = static_cast<ws_header*>(ws);
  ws_header* const rep = report_of(hdr, stream);
  if constexpr (merge_slices_ok<K, V, HAS_V, KeyItA, KeyItB, ValItA, ValItB, KeyOutIt, ValOutIt>::value) {
    using Tuning = merge_slices_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>;
    g.cut(Tuning::TILE);
    const unsigned tiles = (unsigned)g.num_tiles();
    // Up to 8192 tiles (16 M outputs) the pass's launches overlap the kernels before them (8 M pairs sorted in 0.47 ms
    // against 0.51); beyond, waiting CTAs only take slots from running ones (2^26 pairs 4.53 ms against 4.35).
    const bool overlap = tiles <= 8192;
    // Up to 2048 tiles (4 M outputs) of a sort's pass the tiles find their splits themselves, with a launch less (1 M pairs sorted in 120 us
    // against 145, 3 M 207 against 222; 8 M 500 against 484: many CTAs per SM then wait for their searches).
    const bool own_splits = g.run != 0 && tiles <= 2048;
    if (own_splits) a_split = nullptr;
    const cudaError_t e = own_splits ? cudaSuccess : merge_split_async<K, Comp, Tuning::TILE>(ka, kb, g, tiles, comp, a_split, overlap, stream);
    if (e != cudaSuccess) return e;
    if (overlap) {
      timed_launch tl(KID_MERGE, stream);
      const cudaError_t le = launch_after(merge_slices_kernel<K, V, HAS_V, Comp>, tiles, MERGE_BLOCK, 0, stream, ka, kb, va, vb, ko, vo, g, comp,
                                          (const size_t*)a_split, &rep->error);
      log_launch("merge_slices_kernel", tiles, MERGE_BLOCK, 0, g.n, stream);
      return reported(le, rep, hdr);
    }
    timed_launch tl(KID_MERGE, stream);
    merge_slices_kernel<K, V, HAS_V, Comp><<<tiles, MERGE_BLOCK, 0, stream>>>(ka, kb, va, vb, ko, vo, g, comp, a_split, &rep->error);
    log_launch("merge_slices_kernel", tiles, MERGE_BLOCK, 0, g.n, stream);
    return reported(cudaGetLastError(), rep, hdr);
  } else {
  g.cut(TILE);
  const size_t tiles = g.num_tiles();
  merge_partition_kernel<KeyItA, KeyItB, Comp, TILE><<<(unsigned)((tiles + 255) / 256), 256, 0, stream>>>(ka, kb, g, tiles, comp, a_split);
  timed_launch tl(KID_MERGE, stream);
  merge_kernel<KeyItA, KeyItB, ValItA, ValItB, KeyOutIt, ValOutIt, K, V, HAS_V, Comp, IPT>
      <<<(unsigned)tiles, MERGE_BLOCK, 0, stream>>>(ka, kb, va, vb, ko, vo, g, comp, a_split, &rep->error);
  log_launch("merge_kernel", tiles, MERGE_BLOCK, 0, g.n, stream);
  return reported(cudaGetLastError(), rep, hdr);
  }
}

// thrust::merge / merge_by_key: A[0,na) and B[0,nb) sorted by comp -> out[0, na+nb).
template <class K, class V, bool HAS_V, class KeyItA, class KeyItB, class ValItA, class ValItB, class KeyOutIt, class ValOutIt, class Comp>
cudaError_t merge_async(KeyItA ka, size_t na, KeyItB kb, size_t nb, ValItA va, ValItB vb, KeyOutIt ko, ValOutIt vo, Comp comp, void* ws,
                        cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(ws, 0, sizeof(ws_header), stream);
#ifdef TB200_TEST_HOOKS
  if (e == cudaSuccess) e = cudaMemsetAsync(&static_cast<ws_header*>(ws)->flags, (int)(test_hook_flags() & 2u), 1, stream);
#endif
  if (e != cudaSuccess) return e;
  return merge_pass_async<K, V, HAS_V>(ka, kb, va, vb, ko, vo, merge_geometry::single(na, nb), comp, ws, stream);
}

// ---------------------------------------------------------------- merge sort
template <int KB, int VB> struct block_sort_tuning {
  // power-of-two friendly tile of 256 * IPT items whose keys (+ a 2-byte index each) fit 44 KB of shared memory
  static constexpr int BLOCK = MERGE_BLOCK;
  static constexpr int FIT = MERGE_SMEM_BUDGET / (BLOCK * (KB + 2));
  static constexpr int IPT = (KB + VB) <= 8 ? TB200_BSORT_IPT8 : (FIT >= 8 ? 8 : FIT >= 4 ? 4 : FIT >= 2 ? 2 : 1);
  // one slot of padding per thread, where static shared memory has room for it (20-byte keys at 8 items: it has not)
  static constexpr int TILE = BLOCK * IPT, SMEM = 48 * 1024;
  // A merge reads one slot past the tile's end at most: the first run of a pair ends a run's length or more in front of it, and a thread goes
  // no more than its own items, which is the shortest run, past that.
  static constexpr int OVER = 1;
  static constexpr int IDX_SLOTS = TILE + OVER;
  static constexpr bool PADDED = IPT >= 8 && (TILE + BLOCK + OVER) * KB + IDX_SLOTS * 2 + 32 <= SMEM;
  static constexpr int SLOTS = TILE + (PADDED ? BLOCK : 0) + OVER;
  static_assert(SLOTS * KB + IDX_SLOTS * 2 <= SMEM, "key too large for the block sort tile (more than 189 bytes)");
};

// What bounds it is shared memory (the pipe is busy 91 % of a large sort's tiles: 122 wavefronts per 32 items before the
// indexes left in 16-byte stores, 113 since): a thread's IPT consecutive items are written and read back in every round, and
// unpadded that is a stride of IPT words, IPT / 2 lanes to a bank.  One slot of padding per IPT items makes the
// stride odd.  Rounds whose pairs of runs lie inside one warp's items need no barrier of the CTA.  The merge takes its next
// item without a branch: two candidates in registers, one load of the side that was taken.  With a branch for either side a
// warp ran both, and a tile took 46 us instead of 20: 1000 (u32, u32) pairs sorted in 24 us (54 before), 100 k in 50 (85), 8 M in
// 431 (484), of them 127 for the tiles (178).  512 threads of 8 items each: 100 k pairs 47 us, 8 M 447.  Payloads kept in shared
// memory instead of fetched by their index: the same.
template <class KeyIt, class ValIt, class KeyOutIt, class ValOutIt, class K, class V, bool HAS_V, class Comp, int IPT>
__global__ void __launch_bounds__((block_sort_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>::BLOCK), sizeof(K) <= 4 ? TB200_BSORT_CTAS8 : 1)
block_sort_kernel(KeyIt keys, ValIt vals, KeyOutIt keys_out, ValOutIt vals_out, size_t n, Comp comp) {
  using Tuning = block_sort_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>;
  constexpr int BLOCK = Tuning::BLOCK, TILE = Tuning::TILE;
  constexpr bool PADDED = Tuning::PADDED;
  constexpr int SLOTS = Tuning::SLOTS;
  static_assert(IPT == Tuning::IPT, "the tile is the tuning's");
  TB200_SHARED_ARRAY(K, s_key, SLOTS);
  __shared__ __align__(16) unsigned short s_idx[Tuning::IDX_SLOTS];
  auto slot = [](unsigned j) { return PADDED ? j + j / IPT : j; };
  grid_dependents_launch();
  const size_t base = (size_t)blockIdx.x * TILE;
  const unsigned tile_n = n - base < TILE ? (unsigned)(n - base) : (unsigned)TILE;

  // ---- coalesced load, then each thread takes IPT consecutive items (the last of a partial tile fewer)
#pragma unroll
  for (int i = 0; i < IPT; ++i) { const unsigned c = threadIdx.x + i * BLOCK; if (c < tile_n) stash(&s_key[slot(c)], (K)keys[base + c]); }
  __syncthreads();
  K k[IPT]; unsigned short idx[IPT];
  const unsigned first = threadIdx.x * IPT, first_slot = slot(first);
  const unsigned mine = first >= tile_n ? 0u : tile_n - first < (unsigned)IPT ? tile_n - first : (unsigned)IPT;
#pragma unroll
  for (int i = 0; i < IPT; ++i) { idx[i] = (unsigned short)(first + i); if ((unsigned)i < mine) k[i] = s_key[first_slot + i]; else k[i] = K(); }
  // ---- odd-even transposition sort of the thread's items (stable: only swaps when strictly out of order)
#pragma unroll
  for (int r = 0; r < IPT; ++r) {
#pragma unroll
    for (int i = r & 1; i + 1 < IPT; i += 2) {
      const bool swap = (unsigned)(i + 1) < mine && comp(k[i + 1], k[i]);
      const K lo = swap ? k[i + 1] : k[i];
      k[i + 1] = swap ? k[i] : k[i + 1];
      k[i] = lo;
      const unsigned short li = swap ? idx[i + 1] : idx[i];
      idx[i + 1] = swap ? idx[i] : idx[i + 1];
      idx[i] = li;
    }
  }
  // the thread's source indexes, in 16-byte stores where they fill one
  auto put_idx = [&] {
    if constexpr (IPT % 8 == 0) {
#pragma unroll
      for (int q = 0; q < IPT / 8; ++q) {
        uint4 w;
        w.x = idx[8 * q] | (unsigned)idx[8 * q + 1] << 16;
        w.y = idx[8 * q + 2] | (unsigned)idx[8 * q + 3] << 16;
        w.z = idx[8 * q + 4] | (unsigned)idx[8 * q + 5] << 16;
        w.w = idx[8 * q + 6] | (unsigned)idx[8 * q + 7] << 16;
        reinterpret_cast<uint4*>(s_idx + first)[q] = w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < IPT; ++i) s_idx[first + i] = idx[i];
    }
  };
  // ---- rounds of pairwise merges in shared memory
  for (unsigned len = IPT; len < (unsigned)TILE; len <<= 1) {
    const bool in_warp = 2 * len <= 32u * IPT;     // both runs are this warp's own items, in this round and the ones before
    if (in_warp && len > (unsigned)IPT) __syncwarp(); else __syncthreads();
#pragma unroll
    for (int i = 0; i < IPT; ++i) stash(&s_key[first_slot + i], k[i]);
    put_idx();
    if (in_warp) __syncwarp(); else __syncthreads();
    const unsigned a0 = first & ~(2 * len - 1), b0 = a0 + len;
    const unsigned an = a0 >= tile_n ? 0u : tile_n - a0 < len ? tile_n - a0 : len, bn = b0 >= tile_n ? 0u : tile_n - b0 < len ? tile_n - b0 : len;
    unsigned d = first - a0;
    if (d > an + bn) d = an + bn;
    // merge path over the two runs (ties take from the left one)
    unsigned lo = d > bn ? d - bn : 0, hi = d < an ? d : an;
    while (lo < hi) {
      const unsigned mid = (lo + hi) >> 1;
      if (!comp(s_key[slot(b0 + d - 1 - mid)], s_key[slot(a0 + mid)])) lo = mid + 1; else hi = mid;
    }
    unsigned ai = a0 + lo, bi = b0 + (d - lo);
    const unsigned a_end = a0 + an, b_end = b0 + bn;
    // the two candidates stay in registers; only the side that was taken is read again, always: past a run's end that is some
    // slot of the tile which nothing looks at
    K key_a = K(), key_b = K();
    if (std::is_trivially_copyable<K>::value || ai < a_end) key_a = s_key[slot(ai)];
    if (std::is_trivially_copyable<K>::value || bi < b_end) key_b = s_key[slot(bi)];
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const bool take_b = bi < b_end && (ai >= a_end || comp(key_b, key_a));
      idx[i] = s_idx[take_b ? bi : ai];
      k[i] = take_b ? key_b : key_a;
      ai += take_b ? 0u : 1u;
      bi += take_b ? 1u : 0u;
      if (std::is_trivially_copyable<K>::value || (take_b ? bi < b_end : ai < a_end)) {
        const K next = s_key[slot(take_b ? bi : ai)];
        key_b = take_b ? next : key_b;
        key_a = take_b ? key_a : next;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < IPT; ++i) stash(&s_key[first_slot + i], k[i]);
  put_idx();
  __syncthreads();
  // gather the payloads by source index before anything is written: the output may be the input
  [[maybe_unused]] V v_out[HAS_V ? IPT : 1];
  if constexpr (HAS_V) {
#pragma unroll
    for (int i = 0; i < IPT; ++i) { const unsigned c = threadIdx.x + i * BLOCK; if (c < tile_n) v_out[i] = vals[base + s_idx[c]]; }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const unsigned c = threadIdx.x + i * BLOCK;
    if (c < tile_n) {
      keys_out[base + c] = s_key[slot(c)];
      if constexpr (HAS_V) vals_out[base + c] = v_out[i];
    }
  }
}

template <class K, class V, bool HAS_V> constexpr int block_sort_tile_items() { return block_sort_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>::TILE; }

template <class K, class V, bool HAS_V> size_t merge_sort_workspace_bytes(size_t n) { return merge_workspace_bytes<K, V, HAS_V>(n); }

// Stable merge sort of keys (and values) in place; keys_alt / vals_alt are same-sized scratch.
template <class K, class V, bool HAS_V, class Comp>
cudaError_t merge_sort_async(K* keys, K* keys_alt, V* vals, V* vals_alt, size_t n, Comp comp, void* ws, cudaStream_t stream) {
  constexpr int BS_IPT = block_sort_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>::IPT;
  using Tuning = block_sort_tuning<sizeof(K), HAS_V ? sizeof(V) : 0>;
  constexpr size_t BS_TILE = (size_t)Tuning::TILE;
  cudaError_t e = cudaMemsetAsync(ws, 0, sizeof(ws_header), stream);
  if (e != cudaSuccess || n <= 1) return e;
  const size_t tiles = (n + BS_TILE - 1) / BS_TILE;
  int passes = 0;
  for (size_t run = BS_TILE; run < n; run <<= 1) ++passes;
  // the block sort writes to whichever buffer makes the last merge pass land in `keys`
  K* cur_k = (passes & 1) ? keys_alt : keys;
  V* cur_v = (passes & 1) ? vals_alt : vals;
  K* oth_k = (passes & 1) ? keys : keys_alt;
  V* oth_v = (passes & 1) ? vals : vals_alt;
  { timed_launch tl(KID_BLOCK_SORT, stream);
  block_sort_kernel<const K*, const V*, K*, V*, K, V, HAS_V, Comp, BS_IPT><<<(unsigned)tiles, Tuning::BLOCK, 0, stream>>>(keys, vals, cur_k, cur_v, n, comp); }
  log_launch("block_sort_kernel", tiles, Tuning::BLOCK, 0, n, stream);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  for (size_t run = BS_TILE; run < n; run <<= 1) {
    e = merge_pass_async<K, V, HAS_V>((const K*)cur_k, (const K*)cur_k, (const V*)cur_v, (const V*)cur_v, oth_k, oth_v,
                                      merge_geometry::pairwise(n, run), comp, ws, stream);
    if (e != cudaSuccess) return e;
    K* tk = cur_k; cur_k = oth_k; oth_k = tk;
    V* tv = cur_v; cur_v = oth_v; oth_v = tv;
  }
  return cudaSuccess;
}

}  // namespace tb200
