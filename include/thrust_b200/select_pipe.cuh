// Stream compaction of large contiguous inputs on sm_100a on the tile pipeline (tile_pipe.cuh): copy_if,
// partition_copy, the in-place partition and unique_copy, for 4- and 8-byte arithmetic types.
//
// The compute warps count what their part of a tile keeps some tiles ahead and hold its flags in a register (the in-place partition
// finds them again); once the number of items kept before the tile is known they compact their part in place --
// kept items first, dropped ones in a second round --, shifted so that 16-byte pieces in shared memory are
// 16-byte pieces of the output, and store it with one 16-byte store per lane.  The input is read from HBM once.
//
// In-place partition: a tile's carry is known only after every earlier tile has been summarised, so after
// all of them lie in shared memory; the kept items' places (never behind the tile's own end) can then be
// overwritten.  A carry must order those stores behind the other CTAs' copies of what lay there (the pipeline's ORDERED
// form): with released and acquired descriptors the two kernels take 376 us at 2^27 int32, with relaxed ones 357, with
// fences around relaxed ones 396.  Only the dropped items take a trip through scratch memory (partition_rejects_kernel).
//
// Measured on B200, 2^28 int32, half of the items kept (unique: a quarter), against two streaming passes that read
// the input twice / one pass with look-back: copy_if 0.343 ms against 0.460 / 0.613, partition_copy 0.478 against
// 0.645 / 0.804, unique_copy 0.322 against 0.418 / 0.600, partition in place 0.64 against 0.97 (before its descriptors were ordered).  copy_if and
// unique run at 4700 and 4200 GB/s of algorithmic traffic: the warps' chains of shuffles and shared-memory trips are
// what is left (a copy of the same bytes 0.25 and 0.21 ms).  Flags held from count to compaction instead of found twice: 2^27 int32 unique
// 174 -> 150 us, copy_if 177 -> 166.
#pragma once
#include "tile_pipe.cuh"

namespace tb200 {

// where dropped items go: nowhere; a second array, in input order
enum : int { SELECT_DROP = 0, SELECT_SECOND_ARRAY = 1 };

template <class T> using select_parts = pipe_parts<T, PIPE_ROWS * 512 / (int)sizeof(T)>;

// IN_PLACE: out_sel is the input
template <bool UNIQUE, int REJ, bool IN_PLACE, class T, class Pred>
__global__ void __launch_bounds__(PIPE_BLOCK, 1)
select_pipe_kernel(const T* in, T* out_sel, T* out_rej, size_t n, unsigned tiles, Pred pred, tile_chain<unsigned long long, plus_op> chain, ws_header* hdr,
                   ws_header* rep, unsigned long long* d_count) {
  using C = unsigned long long;
  constexpr int VEC = 16 / sizeof(T);
  constexpr int ITEMS = PIPE_TILE_BYTES / sizeof(T);
  constexpr int CHUNK = ITEMS / PIPE_WARPS;
  extern __shared__ __align__(128) unsigned char pipe_raw[];
  using Parts = select_parts<T>;
  __shared__ pipe_state<unsigned, C> st;
  __shared__ __align__(16) vec16 s_edge[UNIQUE ? PIPE_STAGES : 1];   // the 16 bytes in front of the stage's tile
  unsigned char* const stages = pipe_align(pipe_raw);
  pipe_init(st);
  const int lane = lane_id(), warp = threadIdx.x >> 5;

  if (warp == PIPE_LOADER) {
    const unsigned long long policy = l2_stream_policy();
    pipe_loader(st, tiles, &rep->error, [&](unsigned s, unsigned tile) {
      unsigned char* const stage = stages + (size_t)s * Parts::BYTES;
      const size_t base = (size_t)tile * ITEMS;
      Parts::ragged(stage, in + base, n - base);
      __syncwarp();
      if (lane == 0) {
        const unsigned front = UNIQUE && tile > 0 ? 16u : 0u;
        mbar_arrive_expect(&st.full[s], Parts::bytes(n - base) + front);
        if (front) bulk_load(&s_edge[UNIQUE ? s : 0], in + base - VEC, front, &st.full[s], policy);
      }
      __syncwarp();
      if (lane < PIPE_WARPS) Parts::copy(stage, in + base, n - base, lane, &st.full[s], policy);
    });
  } else if (warp == PIPE_PUBLISHER) {
    pipe_publisher<IN_PLACE>(st, chain, tiles, &rep->error, [&](unsigned part) { return (C)__reduce_add_sync(FULL_MASK, lane < PIPE_WARPS ? part : 0u); });
  } else if (warp == PIPE_FOLDER) {
    pipe_folder<IN_PLACE>(st, chain, tiles, (C)0, &rep->error, [&](C total) { hdr->count = rep->count = total; if (d_count) *d_count = total; });
  } else {
    const int mine = warp % PIPE_WARPS;
    // UNIQUE: the item in front of the stage's tile, for its first warp.  Nothing lies in front of the input: its first item is
    // then compared with itself (and kept whatever comes out), because `pred` may only ever see items of the input
    auto tile_front = [&](unsigned s, unsigned tile) {
      return tile > 0 ? reinterpret_cast<const T*>(&s_edge[UNIQUE ? s : 0])[VEC - 1] : Parts::part(stages + (size_t)s * Parts::BYTES, 0)[0];
    };
    // this lane's items of the warp's part and their keep flags, bit v * VEC + k
    static_assert(PIPE_ROWS * VEC <= 32, "a lane's flags fit a word");
    open_words flags;
    auto load_items = [&](unsigned s, T (&x)[PIPE_ROWS][VEC]) {
      const T* part = Parts::part(stages + (size_t)s * Parts::BYTES, mine);
#pragma unroll
      for (int v = 0; v < PIPE_ROWS; ++v) {
        const vec16 r = reinterpret_cast<const vec16*>(part)[v * 32 + lane];
        const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
        for (int k = 0; k < VEC; ++k) x[v][k] = e[k];
      }
    };
    auto flags_of = [&](unsigned tile, const T& edge, const T (&x)[PIPE_ROWS][VEC]) {
      const size_t first = (size_t)tile * ITEMS + (size_t)mine * CHUNK;
      unsigned bits = 0;
      auto scan_flags = [&](auto whole_tag) {
        constexpr bool WHOLE = decltype(whole_tag)::value;   // else only items inside the input are looked at
#pragma unroll
        for (int v = 0; v < PIPE_ROWS; ++v) {
          // UNIQUE: predecessor of the lane's first item of the row: the previous lane's last one, the previous row's, or
          // for the warp's very first item `edge`, the one in front of its part
          T prev = T();
          if constexpr (UNIQUE) {
            prev = shfl_up(x[v][VEC - 1], 1);
            const T wrap = v > 0 ? shfl_idx(x[v > 0 ? v - 1 : 0][VEC - 1], 31) : edge;
            if (lane == 0) prev = wrap;
          }
#pragma unroll
          for (int k = 0; k < VEC; ++k) {
            if (WHOLE || first + (size_t)(v * 32 + lane) * VEC + k < n) {
              bool keep;
              if constexpr (UNIQUE) keep = !pred(k == 0 ? prev : x[v][k > 0 ? k - 1 : 0], x[v][k]); else keep = pred(x[v][k]);
              if (keep) bits |= 1u << (v * VEC + k);
            }
          }
        }
      };
      if (first + CHUNK <= n) scan_flags(std::true_type()); else scan_flags(std::false_type());
      if (UNIQUE && first == 0 && lane == 0) bits |= 1u;   // the input's first item is kept
      return bits;
    };
    pipe_compute<true>(st, tiles, &rep->error,
      [&](unsigned s, unsigned tile) {
        T x[PIPE_ROWS][VEC];
        T edge = T();
        if constexpr (UNIQUE) {
          // nobody compacts its part of this tile before every warp has been here
          edge = mine > 0 ? Parts::part(stages + (size_t)s * Parts::BYTES, mine > 0 ? mine - 1 : 0)[CHUNK - 1] : tile_front(s, tile);
        }
        load_items(s, x);
        const unsigned bits = flags_of(tile, edge, x);
        if constexpr (!IN_PLACE) flags.put(bits);
        return __reduce_add_sync(FULL_MASK, (unsigned)__popc(bits));
      },
      [&](unsigned s, unsigned tile) {
        T x[PIPE_ROWS][VEC];
        load_items(s, x);
        // In place, where a store may hit what another tile is read from, the flags are those of the items as they are now, and
        // what they keep is checked against the count below (2^27 int32: kernel 267 to 269 us, 264 to 265 with held flags and no such check).
        const unsigned bits = IN_PLACE ? flags_of(tile, T(), x) : flags.take();
        T* const buf = Parts::part(stages + (size_t)s * Parts::BYTES, mine);
        __syncwarp();   // every lane has its items: the part may be overwritten
        // kept items before this lane in each row: a scan over the lanes carries four rows' counts, a byte each
        // (a row has at most 128 items)
        static_assert(PIPE_ROWS % 4 == 0 && 32 * VEC <= 255, "a row's count fits a byte");
        unsigned excl[PIPE_ROWS / 4], totals[PIPE_ROWS / 4];
#pragma unroll
        for (int q = 0; q < PIPE_ROWS / 4; ++q) {
          unsigned packed = 0;
#pragma unroll
          for (int v = 0; v < 4; ++v) packed |= (unsigned)__popc((bits >> ((q * 4 + v) * VEC)) & ((1u << VEC) - 1)) << (8 * v);
          const unsigned incl = warp_inclusive_scan(packed, plus_op());
          totals[q] = __shfl_sync(FULL_MASK, incl, 31);
          excl[q] = incl - packed;
        }
        const unsigned before = __reduce_add_sync(FULL_MASK, lane < mine ? st.part[s][lane & (PIPE_WARPS - 1)] : 0u);   // the warps before this one
        const C kept0 = st.carry[s] + before;      // kept items in front of this warp's part
        const size_t first = (size_t)tile * ITEMS + (size_t)mine * CHUNK;
        const unsigned part_n = first >= n ? 0u : n - first < (size_t)CHUNK ? (unsigned)(n - first) : (unsigned)CHUNK;
        unsigned row_off = 0;
#pragma unroll
        for (int q = 0; q < PIPE_ROWS / 4; ++q) row_off += (totals[q] & 255) + ((totals[q] >> 8) & 255) + ((totals[q] >> 16) & 255) + (totals[q] >> 24);
        // What is stored lies inside the output and is what was counted, else it is reported and nothing is stored: the flags held are
        // those of this stage and the carry leaves room.
        if (row_off != st.part[s][mine] || kept0 > first || row_off > part_n) {
          if (lane == 0) record_error(&rep->error, ERR_INCONSISTENT);
          return;
        }
        T* const dst = out_sel + kept0;
        const unsigned shift = run_shift(dst);
        row_off = 0;
#pragma unroll
        for (int v = 0; v < PIPE_ROWS; ++v) {
          unsigned r = shift + row_off + ((excl[v / 4] >> (8 * (v % 4))) & 255);
#pragma unroll
          for (int k = 0; k < VEC; ++k) {
            const bool keep = (bits >> (v * VEC + k)) & 1;
            if (keep) buf[r] = x[v][k];
            r += keep;
          }
          row_off += (totals[v / 4] >> (8 * (v % 4))) & 255;
        }
        __syncwarp();
        warp_store_run(dst - shift, buf, shift, shift + row_off);
        if constexpr (REJ != SELECT_DROP) {
          const unsigned kept = row_off;
          T* const rdst = out_rej + (first - (size_t)kept0);
          const unsigned rshift = run_shift(rdst);
          __syncwarp();
          row_off = 0;
#pragma unroll
          for (int v = 0; v < PIPE_ROWS; ++v) {
            // dropped items before this lane in the row: its first index in the row less the kept ones
            unsigned r = rshift + row_off + lane * VEC - ((excl[v / 4] >> (8 * (v % 4))) & 255);
#pragma unroll
            for (int k = 0; k < VEC; ++k) {
              const bool drop = !((bits >> (v * VEC + k)) & 1);
              if (drop && (unsigned)(v * 32 + lane) * VEC + k < part_n) buf[r] = x[v][k];
              r += drop;
            }
            row_off += 32 * VEC - ((totals[v / 4] >> (8 * (v % 4))) & 255);
          }
          __syncwarp();
          if (part_n) warp_store_run(rdst - rshift, buf, rshift, rshift + part_n - kept);
        }
      });
  }
}

// Second half of the in-place partition: the dropped items, in input order in `rejects`, go behind the
// hdr->count kept ones.  16-byte loads and, shifted inside a warp, 16-byte stores.
template <class T>
__global__ void __launch_bounds__(256)
partition_rejects_kernel(T* data, const T* rejects, size_t n, const ws_header* hdr) {
  constexpr int VEC = 16 / sizeof(T);
  const size_t kept = (size_t)hdr->count;
  if (kept > n) return;
  const size_t count = n - kept;
  T* const dst = data + kept;
  const size_t head = ((16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15) / sizeof(T);   // items in front of dst's first 16-byte boundary
  const size_t tid = (size_t)blockIdx.x * 256 + threadIdx.x, stride = (size_t)gridDim.x * 256;
  if (count <= head) { if (tid < count) dst[tid] = rejects[tid]; return; }
  if (tid < head) dst[tid] = rejects[tid];
  const size_t nvec = (count - head) / VEC;
  constexpr int U = 4;
  for (size_t v0 = tid; v0 < nvec; v0 += U * stride) {
    vec16 r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t v = v0 + u * stride;
      if (v < nvec) {
        T* e = reinterpret_cast<T*>(&r[u]);
#pragma unroll
        for (int k = 0; k < VEC; ++k) e[k] = __ldcs(rejects + head + v * VEC + k);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) { const size_t v = v0 + u * stride; if (v < nvec) store_stream16(dst + head + v * VEC, r[u]); }
  }
  const size_t done = head + nvec * VEC;
  if (done + tid < count) dst[done + tid] = rejects[done + tid];
}

template <class T> constexpr size_t select_pipe_tile_items() { return PIPE_TILE_BYTES / sizeof(T); }
template <class T> size_t select_pipe_workspace_bytes(size_t n) {
  return sizeof(ws_header) + tile_chain<unsigned long long, plus_op>::bytes((n + select_pipe_tile_items<T>() - 1) / select_pipe_tile_items<T>());
}

// Launches the pipeline compaction if the device can hold it and takes the launch (launched = true).  `in` is 16-byte aligned.
template <bool UNIQUE, int REJ, bool IN_PLACE, class T, class Pred>
cudaError_t select_pipe_launch(const T* in, T* out_sel, T* out_rej, size_t n, Pred pred, unsigned long long* d_count, void* ws, cudaStream_t stream, bool& launched) {
  launched = false;
  const size_t tiles = (n + select_pipe_tile_items<T>() - 1) / select_pipe_tile_items<T>();
  if (tiles >= 0xffffff00ull || n == 0) return cudaSuccess;
  static thread_local bool ready[64] = {false};
  auto kern = select_pipe_kernel<UNIQUE, REJ, IN_PLACE, T, Pred>;
  const size_t smem = pipe_smem_bytes(select_parts<T>::BYTES, 0);
  const size_t grid = pipe_grid(kern, smem, tiles, ready);
  if (grid == 0) return cudaSuccess;
  char* base = static_cast<char*>(ws);
  ws_header* hdr = reinterpret_cast<ws_header*>(base);
  tile_chain<unsigned long long, plus_op> chain;
  chain.bind(base + sizeof(ws_header), tiles);
  cudaError_t e = pipe_clear(base, sizeof(ws_header) + tile_chain<unsigned long long, plus_op>::bytes(tiles), stream);
  if (e != cudaSuccess) return e;
  timed_launch tl(KID_SELECT, stream);
  ws_header* const rep = report_of(hdr, stream);
  e = pipe_launch(kern, grid, smem, stream, in, out_sel, out_rej, n, (unsigned)tiles, pred, chain, hdr, rep, d_count);
  if (launch_refused(e)) return cudaSuccess;
  reported(e, rep, hdr);
  launched = true;
  log_launch("select_pipe_kernel", grid, PIPE_BLOCK, smem, n, stream);
  return e;
}

}  // namespace tb200
