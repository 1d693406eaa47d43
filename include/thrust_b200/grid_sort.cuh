// Radix sort of inputs that fit the registers of the chip's CTAs (up to 448 k items, 288 k with 8-byte keys), in one cooperative launch.
//
// Between the cluster sort (cluster_sort.cuh: up to 16 SMs) and the general one (radix_sort.cuh: a chain of launches with look-backs between
// tiles) lies a range where a digit place is latency, not work.  Here every CTA keeps its share of the items in registers;
// a digit place is
//   rank      every warp ranks its rows on private counters, the CTA stacks them, stores its 256 counts in a table in
//             global memory and puts its items in digit order in shared memory;
//   meeting   of all CTAs, at a counter (bounded wait);
//   place     every CTA adds the table up (before it, in all), and stores its items, consecutive lanes mostly to consecutive
//             places, where they belong in the input's own array -- every CTA holds its items, nothing there is needed any more;
//   meeting   after which every CTA reads its share back, past its L1 cache.
// A digit place that all keys share is left out, as in the general sort.  Same order, same stability.
#pragma once
#include "cluster_sort.cuh"
#include "common.cuh"
#include "radix_keys.cuh"

namespace tb200 {

constexpr int GSORT_BLOCK = 512;
constexpr int GSORT_PARTS = GSORT_BLOCK / (RADIX_BINS / 2);   // in which the CTAs' counts are added up
// Counts that a thread has in flight, the last ones of the table too: one after the other those past a multiple of 32 CTAs cost up to 1 us a
// digit place (microseconds, now / so: u64 50 k 61 / 67, 114 k 69 / 74, 300 k 80 / 87; f32 37 / 40, 41 / 43, 44 / 47; with every batch checked
// for the table's end up to 1 us more again).
constexpr int GSORT_BATCH = 8;

template <class Item, int IPT> constexpr size_t gsort_smem_bytes() {
  return (size_t)GSORT_BLOCK * IPT * sizeof(Item) + (GSORT_BLOCK / 32) * RADIX_BINS * 4 + 2 * GSORT_PARTS * RADIX_BINS * 4;
}
// the CTAs' digit counts, for two digit places in turn
inline size_t gsort_table_bytes(size_t ctas) { return 2 * ctas * RADIX_BINS * sizeof(unsigned short); }

// A meeting of all CTAs of a resident grid at a counter that starts at zero.  When a wait runs out the CTA goes on: what it then
// computes is wrong, but every access stays inside the arrays.
struct grid_meeting {
  unsigned* counter; unsigned* err;
  unsigned met = 0;
  bool gave_up = false;   // then it does not wait again
  __device__ __forceinline__ void operator()() {
    __syncthreads();
    met += gridDim.x;
    if (threadIdx.x == 0) {
      __threadfence();
#ifdef TB200_TEST_HOOKS
      const bool stays_away = blockIdx.x == 0 && (reinterpret_cast<const ws_header*>(err)->flags & 1u);   // err points at the header's first word
      if (!stays_away)
#endif
      atomicAdd(counter, 1u);
      unsigned iter = 0;
      while (!gave_up && ld_acquire_u32(counter) < met)
        if (++iter > SPIN_LIMIT) { record_error(err, ERR_LOOKBACK_TIMEOUT); gave_up = true; }
      __threadfence();
    }
    __syncthreads();
  }
};

// rows: rows of 32 items per warp, at most IPT; every CTA holds GSORT_BLOCK * rows places.  table: gsort_table_bytes(gridDim.x).
template <class UK, class UV, bool HAS_V, bool IS_FLOAT, int IPT>
__global__ void __launch_bounds__(GSORT_BLOCK, 1)
grid_sort_kernel(UK* keys, UV* vals, unsigned n, unsigned rows, key_coding coding, int first_pass, int num_passes, unsigned short* table, ws_header* hdr,
                 ws_header* rep) {
  grid_meeting meet{&hdr->ticket, &rep->error};
  using Item = typename csort_item<UK, UV, HAS_V>::type;
  constexpr int NWARPS = GSORT_BLOCK / 32;
  extern __shared__ __align__(16) unsigned char gsort_raw[];
  Item* const s_stage = reinterpret_cast<Item*>(gsort_raw);           // this CTA's items in digit order
  unsigned* const warp_hist = reinterpret_cast<unsigned*>(s_stage + GSORT_BLOCK * IPT);   // [NWARPS][256]
  unsigned* const s_before = warp_hist + NWARPS * RADIX_BINS;         // [GSORT_PARTS][256]: counts of the CTAs before this one
  unsigned* const s_total = s_before + GSORT_PARTS * RADIX_BINS;      // [GSORT_PARTS][256]: of all CTAs
  __shared__ unsigned s_scan[2][RADIX_BINS / 32];
  __shared__ unsigned s_goff[RADIX_BINS];
  const unsigned me = blockIdx.x, ctas = gridDim.x;
  const int lane = lane_id(), warp = threadIdx.x >> 5, t = threadIdx.x;
  const unsigned lanemask_ge = ~((1u << lane) - 1);
  const unsigned chunk = GSORT_BLOCK * rows;
  const unsigned wofs = warp * (32 * rows) + lane;                    // this lane's first item inside the CTA's chunk
  const unsigned base = me * chunk;
  const unsigned mine = base >= n ? 0u : n - base < chunk ? n - base : chunk;
  const unsigned row_pads = (0u - n) & 31u;                           // places past the end in the row that holds the end

  UK key[IPT]; UV val[HAS_V ? IPT : 1];
  auto load = [&] {   // past the L1 cache, which may hold what lay there before
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      const unsigned at = wofs + i * 32;
      const bool in = (unsigned)i < rows && at < mine;
      key[i] = in ? load_cg_any(keys + base + at) : (UK)0;
      if constexpr (HAS_V) val[i] = in ? load_cg_any(vals + base + at) : (UV)0;
    }
  };
  load();
  unsigned* const my_hist = warp_hist + warp * RADIX_BINS;
  const int end_pass = first_pass + num_passes;
  for (int p = first_pass; p < end_pass; ++p) {
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
    unsigned short* const counts = table + (size_t)(p & 1) * ctas * RADIX_BINS;
    const unsigned local = stack_digits<NWARPS>(warp_hist, s_scan[0], [&](unsigned count) { counts[me * RADIX_BINS + t] = (unsigned short)count; });
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
      if ((unsigned)i < rows && wofs + i * 32 < mine) {
        Item it;
        if constexpr (HAS_V) { it.k = key[i]; it.v = val[i]; } else it = key[i];
        s_stage[(pd[i] & 0xffffu) + my_hist[pd[i] >> 16]] = it;
      }
    }
    meet();     // the counts are there, and every CTA holds its items in registers and s_stage
    {
      // the counts of all CTAs: a thread takes two digits (one word) of every GSORT_PARTS-th CTA
      const unsigned part = t / (RADIX_BINS / 2), pair = t % (RADIX_BINS / 2);
      unsigned before0 = 0, before1 = 0, all0 = 0, all1 = 0;
      const unsigned* const words = reinterpret_cast<const unsigned*>(counts) + pair;
      auto add_batch = [&](unsigned first, auto whole_tag) {
        unsigned w[GSORT_BATCH];
#pragma unroll
        for (int b = 0; b < GSORT_BATCH; ++b) {
          const unsigned q = first + b * GSORT_PARTS;
          w[b] = decltype(whole_tag)::value || q < ctas ? __ldcg(words + q * (RADIX_BINS / 2)) : 0u;
        }
#pragma unroll
        for (int b = 0; b < GSORT_BATCH; ++b) {
          const unsigned c0 = w[b] & 0xffffu, c1 = w[b] >> 16;
          if (first + b * GSORT_PARTS < me) { before0 += c0; before1 += c1; }
          all0 += c0; all1 += c1;
        }
      };
      unsigned first = part;
      for (; first + (GSORT_BATCH - 1) * GSORT_PARTS < ctas; first += GSORT_BATCH * GSORT_PARTS) add_batch(first, std::true_type());
      if (first < ctas) add_batch(first, std::false_type());
      s_before[part * RADIX_BINS + 2 * pair] = before0; s_before[part * RADIX_BINS + 2 * pair + 1] = before1;
      s_total[part * RADIX_BINS + 2 * pair] = all0; s_total[part * RADIX_BINS + 2 * pair + 1] = all1;
    }
    __syncthreads();
    unsigned total = 0, before = 0, incl = 0;
    if (t < RADIX_BINS) {
#pragma unroll
      for (int q = 0; q < GSORT_PARTS; ++q) { before += s_before[q * RADIX_BINS + t]; total += s_total[q * RADIX_BINS + t]; }
      incl = warp_inclusive_scan(total, plus_op());
      if (lane == 31) s_scan[1][warp] = incl;
    }
    const bool shared_digit = t < RADIX_BINS && total - (t == RADIX_BINS - 1 ? row_pads : 0u) == n;
    if (__syncthreads_or(shared_digit)) continue;   // every key has this digit: nothing moves
    if (t < RADIX_BINS) {
      unsigned off = incl - total + before - local;   // from this CTA's staged order to the whole one
#pragma unroll
      for (int w = 0; w < RADIX_BINS / 32; ++w) { const unsigned x = s_scan[1][w]; off += w < warp ? x : 0u; }
      s_goff[t] = off;
    }
    __syncthreads();
    for (unsigned j = t; j < mine; j += GSORT_BLOCK) {
      const Item it = s_stage[j];
      UK k;
      if constexpr (HAS_V) k = it.k; else k = it;
      const unsigned pos = s_goff[key_digit<IS_FLOAT>(k, shift, dmask)] + j;
      if (pos < n) {   // always, unless a meeting was given up
        keys[pos] = k;
        if constexpr (HAS_V) vals[pos] = it.v;
      }
    }
    if (p + 1 < end_pass) { meet(); load(); }
  }
}

// CTAs for n items: two rows of 32 per warp while that does, then four, then as many as it takes on all SMs.  Fewer rows are less ranking, fewer
// CTAs a shorter table (microseconds at 100 k f32 keys, 2, 4 and 8 rows: 37, 41, 47; at 262 k, 4, 6 and 8 rows: 41, 49, 48).
inline unsigned gsort_ctas(size_t n) {
  const size_t sms = (size_t)current_device_info().sm_count, row = (size_t)GSORT_BLOCK;
  const size_t rows = n <= sms * row * 2 ? 2 : n <= sms * row * 4 ? 4 : (n + sms * row - 1) / (sms * row);
  return (unsigned)((n + row * rows - 1) / (row * rows));
}
// Up to which input it is the faster route.  A call and the wait for it, microseconds here / on the general route at 160 k, 256 k, 288 k and
// 448 k: u32 + u32 44 / 60, 44 / 62, 46 / 62, 51 / 63; u32 + u64 44 / 58, 46 / 60, 49 / 59, 56 / 62; f32 keys 40 / 61, 42 / 63, 44 / 63, 49 / 64;
// u64 of 64 random bits + u32 80 / 102, 84 / 106, 88 / 106, 98 / 119, of 40 bits 72 / 75, 74 / 77, 80 / 78, 89 / 85.  How many bits vary is
// not known beforehand, so the line of the 8-byte keys lies where the one loses 5 us at most (40 bits, keys alone: 76 / 71) and the other gains 16.
template <int KB, int VB> constexpr size_t gsort_max_items() { return (KB <= 4 ? (size_t)448 : (size_t)288) << 10; }
// Scratch behind the header: the table of as many CTAs as any input of up to n items has here, so that what was asked for a large input
// is enough for every smaller one.
template <int KB, int VB> size_t gsort_workspace_bytes(size_t n) {
  const size_t most = gsort_max_items<KB, VB>(), sms = (size_t)current_device_info().sm_count;
  const size_t of_two_rows = ((n < most ? n : most) + 2 * GSORT_BLOCK - 1) / (2 * GSORT_BLOCK);
  return gsort_table_bytes(of_two_rows < sms ? of_two_rows : sms);
}

// Launches the sort if the input is small enough and the device can hold its CTAs (launched = true).
template <class UK, class UV, bool HAS_V, bool IS_FLOAT, int IPT>
cudaError_t grid_sort_launch(UK* keys, UV* vals, size_t n, unsigned ctas, unsigned rows, key_coding coding, int first_pass, int num_passes, ws_header* hdr,
                             cudaStream_t stream, bool& launched) {
  launched = false;
  constexpr size_t smem = gsort_smem_bytes<typename csort_item<UK, UV, HAS_V>::type, IPT>();
  auto kern = grid_sort_kernel<UK, UV, HAS_V, IS_FLOAT, IPT>;
  static thread_local bool ready[64] = {false};
  int dev = 0;
  if (smem > (size_t)current_device_info().max_smem_optin || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaSuccess;
  if (!ready[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) { cudaGetLastError(); return cudaSuccess; }
    ready[dev] = true;
  }
  cudaError_t e = cudaMemsetAsync(hdr, 0, sizeof(ws_header), stream);
#ifdef TB200_TEST_HOOKS
  if (e == cudaSuccess) e = cudaMemsetAsync(&hdr->flags, (int)(test_hook_flags() & 1u), 1, stream);
#endif
  if (e != cudaSuccess) return e;
  ws_header* const rep = report_of(hdr, stream);
  timed_launch tl(KID_ONESWEEP, stream);
  e = cooperative_launch(kern, ctas, GSORT_BLOCK, smem, stream, keys, vals, (unsigned)n, rows, coding, first_pass, num_passes,
                         reinterpret_cast<unsigned short*>(hdr + 1), hdr, rep);
  if (launch_refused(e)) return cudaSuccess;
  reported(e, rep, hdr);
  launched = true;
  log_launch("grid_sort_kernel", ctas, GSORT_BLOCK, smem, n, stream);
  return e;
}

template <class UK, class UV, bool HAS_V>
cudaError_t grid_sort_async(UK* keys, UV* vals, size_t n, key_coding coding, int first_pass, int num_passes, ws_header* hdr, cudaStream_t stream, bool& launched) {
  launched = false;
  if (n > gsort_max_items<sizeof(UK), HAS_V ? sizeof(UV) : 0>()) return cudaSuccess;
  const unsigned ctas = gsort_ctas(n), rows = (unsigned)((n + (size_t)ctas * GSORT_BLOCK - 1) / ((size_t)ctas * GSORT_BLOCK));   // the items spread evenly
  auto go = [&](auto is_float, auto ipt) {
    return grid_sort_launch<UK, UV, HAS_V, decltype(is_float)::value, decltype(ipt)::value>(keys, vals, n, ctas, rows, coding, first_pass, num_passes, hdr, stream, launched);
  };
  auto by_rows = [&](auto is_float) {
    if (rows <= 4) return go(is_float, std::integral_constant<int, 4>());
    if (rows <= 8) return go(is_float, std::integral_constant<int, 8>());
    return cudaSuccess;
  };
  if constexpr (sizeof(UK) >= 4) { if (coding.kind == KEY_FLOAT) return by_rows(std::true_type()); }
  return by_rows(std::false_type());
}

}  // namespace tb200
