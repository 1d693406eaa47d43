// Radix sort of small inputs on sm_100a: the whole sort in one launch, by one thread-block cluster of up to
// 16 CTAs that keeps keys and values in registers and distributed shared memory from the first digit to
// the last.
//
// At these sizes the general sort (radix_sort.cuh) is a chain of dependent launches -- clear, histogram, bucket
// bases, one per digit place, copy back -- each far too small to fill the chip; its time is launch and
// look-back latency, whatever n is.  Here a digit place costs two cluster barriers:
//   rank      every warp ranks its rows on private counters in shared memory (warp_rank, as onesweep_kernel does), the
//             CTA stacks its warps' counts, pushes the 256 sums into every CTA of the cluster and puts its items
//             in digit order in its own shared memory;
//   barrier
//   place     every CTA scans the cluster's counts and stores its items, consecutive lanes to (mostly) consecutive
//             places, in the shared memory of the CTAs that own those places, key and value in one store;
//   barrier, after which every CTA reads its items back in order.
// (Stored straight from the registers in input order, a key and a value at a time, the scattered remote stores
// were two thirds of a pass: about 1.7 cycles each per SM.)  A digit place that all keys share is left out,
// as in the general sort.  Same order, same stability.
//
// Measured on B200, microseconds: f32 keys 22 at 1 k, 26 at 10 k, 30 at 32 k; u32 + u32 23, 30, 36; u64 + u64 35, 44, 58.  csort_max_items says
// where it stops.
#pragma once
#include "cluster.cuh"
#include "common.cuh"
#include "radix_keys.cuh"

namespace tb200 {

constexpr int CSORT_BLOCK = 512;
constexpr int CSORT_MAX_CTAS = CLUSTER_MAX_CTAS;

// What moves between the CTAs: a key alone, or a key and its value in one 8- or 16-byte word.
template <class UK, class UV, bool HAS_V> struct csort_item { using type = UK; };
template <class UK, class UV> struct csort_item<UK, UV, true> {
  struct alignas(sizeof(UK) + sizeof(UV) <= 8 ? 8 : 16) type { UV v; UK k; };
};

// Up to how many items the cluster is the faster route.  Microseconds here / in the grid sort on either side of the lines: keys alone at 32 k,
// 44 k and 56 k: f32 29 / 33, 33 / 35, 37 / 35; u64 53 / 57, 62 / 62, 69 / 61; u16 19 / 21, 22 / 22, 23 / 23; u8 14 / 15, 16 / 15, 16 / 15; u32 + u32 32 / 34,
// 36 / 36, 40 / 36; at 28 k, 32 k and 36 k: u32 + u64 34 / 35, 36 / 35, 39 / 36; u64 + u32 59 / 61, 61 / 61, 68 / 64; u16 + u32 21 / 22, 21 / 22,
// 23 / 23; u64 of which 40 bits vary: alone 55 / 56 at 44 k, with u32 52 / 54 at 32 k.
template <class UK, class UV, bool HAS_V> constexpr size_t csort_max_items() {
  return (size_t)(!HAS_V || (sizeof(UK) == 4 && sizeof(UV) == 4) ? 44 : 32) << 10;
}

template <class Item, int IPT> constexpr size_t csort_smem_bytes() {
  return 2 * (size_t)CSORT_BLOCK * IPT * sizeof(Item) + (CSORT_BLOCK / 32) * RADIX_BINS * 4 + 2 * CSORT_MAX_CTAS * RADIX_BINS * 4;
}

// rows: rows of 32 items per warp, at most IPT; the grid's CTAs hold CSORT_BLOCK * rows places each.
template <class UK, class UV, bool HAS_V, bool IS_FLOAT, int IPT>
__global__ void __launch_bounds__(CSORT_BLOCK, 1)
cluster_sort_kernel(UK* keys, UV* vals, unsigned n, unsigned rows, key_coding coding, int first_pass, int num_passes, ws_header* hdr) {
  using Item = typename csort_item<UK, UV, HAS_V>::type;
  constexpr int NWARPS = CSORT_BLOCK / 32;
  extern __shared__ __align__(16) unsigned char csort_raw[];
  Item* const s_item = reinterpret_cast<Item*>(csort_raw);            // the cluster's items in order, `chunk` per CTA
  Item* const s_stage = s_item + CSORT_BLOCK * IPT;                   // this CTA's items in digit order
  unsigned* const warp_hist = reinterpret_cast<unsigned*>(s_stage + CSORT_BLOCK * IPT);   // [NWARPS][256]
  unsigned* const counts = warp_hist + NWARPS * RADIX_BINS;           // [2][CTAs][256]: every CTA's digit counts, by pass parity
  __shared__ unsigned s_scan[2][RADIX_BINS / 32];
  __shared__ unsigned s_goff[RADIX_BINS];
  const unsigned me = cluster_rank(), ctas = cluster_size();
  const int lane = lane_id(), warp = threadIdx.x >> 5, t = threadIdx.x;
  const unsigned lanemask_ge = ~((1u << lane) - 1);
  const unsigned chunk = CSORT_BLOCK * rows;
  const unsigned wofs = warp * (32 * rows) + lane;                    // this lane's first item inside the CTA's chunk
  const unsigned base = me * chunk;
  const unsigned mine = base >= n ? 0u : n - base < chunk ? n - base : chunk;
  const unsigned row_pads = (0u - n) & 31u;                           // places past the end in the row that holds the end
  if (me == 0 && t < (int)(sizeof(ws_header) / 4)) reinterpret_cast<unsigned*>(hdr)[t] = 0;

  UK key[IPT]; UV val[HAS_V ? IPT : 1];
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const unsigned at = wofs + i * 32;
    const bool in = (unsigned)i < rows && at < mine;
    key[i] = in ? keys[base + at] : (UK)0;
    if constexpr (HAS_V) val[i] = in ? vals[base + at] : (UV)0;
  }
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // every CTA has started before another one stores into it
  bool started = false;
  unsigned* const my_hist = warp_hist + warp * RADIX_BINS;
  unsigned parity = 0;
  for (int p = first_pass; p < first_pass + num_passes; ++p, parity ^= 1) {
    const int shift = p * RADIX_BITS;
    const unsigned dmask = digit_mask<UK>(coding, shift);
#pragma unroll
    for (int q = 0; q < RADIX_BINS / 32; ++q) my_hist[q * 32 + lane] = 0;   // only this warp uses them until the stacking
    __syncwarp();
    unsigned pd[IPT];   // low 16 bits: rank inside the warp, then the digit
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      if ((unsigned)i < rows && warp * (32 * rows) + i * 32 < mine) {       // the row holds items
        // places past the end in the input's last row hold the highest digit and rank last
        const unsigned d = wofs + i * 32 < mine ? key_digit<IS_FLOAT>(key[i], shift, dmask) : (unsigned)(RADIX_BINS - 1);
        pd[i] = warp_rank<RADIX_BITS>(my_hist, d, lanemask_ge) | (d << 16);
      }
    }
    __syncthreads();
    if (!started) { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); started = true; }
    unsigned* const table = counts + parity * (CSORT_MAX_CTAS * RADIX_BINS);
    const unsigned local = stack_digits<NWARPS>(warp_hist, s_scan[0], [&](unsigned count) {
      const unsigned at = smem_addr(table + me * RADIX_BINS + t);
      for (unsigned q = 0; q < ctas; ++q) cluster_store(cluster_addr(at, q), count);
    });
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      if ((unsigned)i < rows && wofs + i * 32 < mine) {
        Item it;
        if constexpr (HAS_V) { it.k = key[i]; it.v = val[i]; } else it = key[i];
        s_stage[(pd[i] & 0xffffu) + my_hist[pd[i] >> 16]] = it;
      }
    }
    cluster_barrier();     // the tables are complete, and every CTA holds its items in registers and s_stage
    unsigned total = 0, before = 0, incl = 0;
    if (t < RADIX_BINS) {
#pragma unroll 4
      for (unsigned q = 0; q < ctas; ++q) { const unsigned c = table[q * RADIX_BINS + t]; if (q < me) before += c; total += c; }
      incl = warp_inclusive_scan(total, plus_op());
      if (lane == 31) s_scan[1][warp] = incl;
    }
    const bool shared_digit = t < RADIX_BINS && total - (t == RADIX_BINS - 1 ? row_pads : 0u) == n;
    if (__syncthreads_or(shared_digit)) continue;   // every key has this digit: nothing moves
    if (t < RADIX_BINS) {
      unsigned off = incl - total + before - local;   // from this CTA's staged order to the cluster's
#pragma unroll
      for (int w = 0; w < RADIX_BINS / 32; ++w) { const unsigned x = s_scan[1][w]; off += w < warp ? x : 0u; }
      s_goff[t] = off;
    }
    __syncthreads();
    for (unsigned j = t; j < mine; j += CSORT_BLOCK) {
      const Item it = s_stage[j];
      UK k;
      if constexpr (HAS_V) k = it.k; else k = it;
      const unsigned pos = s_goff[key_digit<IS_FLOAT>(k, shift, dmask)] + j;
      const unsigned cta = pos / chunk, at = pos - cta * chunk;
      cluster_store(cluster_addr(smem_addr(s_item + at), cta), it);
    }
    cluster_barrier();
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      if ((unsigned)i < rows && wofs + i * 32 < mine) {
        const Item it = s_item[wofs + i * 32];
        if constexpr (HAS_V) { key[i] = it.k; val[i] = it.v; } else key[i] = it;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < IPT; ++i) {
    const unsigned at = wofs + i * 32;
    if ((unsigned)i < rows && at < mine) {
      keys[base + at] = key[i];
      if constexpr (HAS_V) vals[base + at] = val[i];
    }
  }
}

// Launches the cluster sort if the input is small enough and the device can hold the cluster (launched = true).
template <class UK, class UV, bool HAS_V, bool IS_FLOAT, int IPT>
cudaError_t cluster_sort_launch(UK* keys, UV* vals, size_t n, key_coding coding, int first_pass, int num_passes, ws_header* hdr, cudaStream_t stream, bool& launched) {
  launched = false;
  constexpr size_t smem = csort_smem_bytes<typename csort_item<UK, UV, HAS_V>::type, IPT>();
  auto kern = cluster_sort_kernel<UK, UV, HAS_V, IS_FLOAT, IPT>;
  unsigned ctas = 1;
  while (ctas * (size_t)CSORT_BLOCK * IPT < n) ctas <<= 1;
  if (ctas > (unsigned)CSORT_MAX_CTAS) return cudaSuccess;
  const unsigned rows = (unsigned)((n + (size_t)ctas * CSORT_BLOCK - 1) / ((size_t)ctas * CSORT_BLOCK));   // the items spread evenly
  static thread_local unsigned largest[64] = {0};
  timed_launch tl(KID_ONESWEEP, stream);
  const cudaError_t e = cluster_launch(kern, ctas, CSORT_BLOCK, smem, stream, largest, launched, keys, vals, (unsigned)n, rows, coding, first_pass, num_passes, hdr);
  if (!launched) return e;
  reported(e, report_of(hdr, stream), hdr);   // nothing to report: no wait of this kernel runs out
  log_launch("cluster_sort_kernel", ctas, CSORT_BLOCK, smem, n, stream);
  return e;
}

template <class UK, class UV, bool HAS_V>
cudaError_t cluster_sort_async(UK* keys, UV* vals, size_t n, key_coding coding, int first_pass, int num_passes, ws_header* hdr, cudaStream_t stream, bool& launched) {
  launched = false;
  constexpr size_t MOST = csort_max_items<UK, UV, HAS_V>(), ROW = (size_t)CSORT_BLOCK * CSORT_MAX_CTAS;
  if (n > MOST) return cudaSuccess;
  auto go = [&](auto is_float, auto ipt) {
    return cluster_sort_launch<UK, UV, HAS_V, decltype(is_float)::value, decltype(ipt)::value>(keys, vals, n, coding, first_pass, num_passes, hdr, stream, launched);
  };
  auto by_rows = [&](auto is_float) {
    if constexpr (MOST > 4 * ROW) { if (n > 4 * ROW) return go(is_float, std::integral_constant<int, 6>()); }
    return go(is_float, std::integral_constant<int, 4>());
  };
  static_assert(MOST <= 6 * ROW, "rows of the largest cluster");
  if constexpr (sizeof(UK) >= 4) { if (coding.kind == KEY_FLOAT) return by_rows(std::true_type()); }
  return by_rows(std::false_type());
}

}  // namespace tb200
