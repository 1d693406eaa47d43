// Inclusive / exclusive scan for sm_100a.  Large contiguous inputs under plus, min or max go to the tile
// pipeline (scan_pipe.cuh).  This file holds the single-pass kernel with decoupled look-back that serves
// any operator, any iterator and small inputs, the windowed kernel for large inputs behind an iterator
// (a transform_iterator, say) and the dispatch.
//
// Single pass:
// One CTA per tile; tiles are handed out by an atomic ticket so that a tile's predecessors have
// always started.  Each lane of a warp loads 16-byte vectors lane-interleaved (a warp instruction
// touches 512 contiguous bytes), scans its vectors in registers, the warp scans each row of
// vector totals with shuffles, and warp 0 resolves the tile's prefix by looking back over the
// preceding tiles' published aggregates.  The output is written with the same 16-byte pattern,
// so every element is read once and written once: 2 * sizeof(T) bytes of HBM traffic per element.
// An input of up to 16 tiles is one cluster's, a tile per CTA: nothing to clear, no ticket, no look-back (a call and the wait for it: 50 k
// int32 11.4 us against 13.4, 131 k 11.5 against 14.0, 65 k doubles 12.2 against 14.9).
// Replaces the cub::DispatchScan call of thrust/system/cuda/detail/scan.h:61-114 and :139-192.
#pragma once
#include "common.cuh"
#include "cluster.cuh"
#include "reduce.cuh"
#include "scan_pipe.cuh"

namespace tb200 {

constexpr int SCAN_BLOCK = 256;
// Bytes of input per thread.  Measured on B200 at 2^28 int32: 64 B -> 0.75 ms, 128 B -> 0.62 ms; the
// kernel is bound by the wait for the preceding tiles' prefixes, which shrinks with the number of
// tiles in flight, so fewer and larger tiles win.
constexpr int SCAN_BYTES_PER_THREAD = 128;

template <class T> struct scan_tuning {
  static constexpr int IPT = sizeof(T) >= 32 ? 4 : (int)(SCAN_BYTES_PER_THREAD / sizeof(T));
};

template <class InIt, class OutIt, class T, class Op, bool INCLUSIVE, int VEC, int IPT>
__global__ void __launch_bounds__(SCAN_BLOCK, 4)
scan_kernel(InIt in, OutIt out, size_t n, T init, bool has_init, const T* init_ptr, Op op, tile_state<T> ts, ws_header* hdr, ws_header* rep,
            bool one_cluster) {
  if (one_cluster && gridDim.x > 1) cluster_arrive_started();
  if (init_ptr) { init = *init_ptr; has_init = true; }   // an initial value that lives on the device (the carry of a sharded scan)
  constexpr int VPT = IPT / VEC;
  constexpr int NWARPS = SCAN_BLOCK / 32;
  constexpr int WCHUNK = 32 * IPT;
  constexpr size_t TILE = (size_t)SCAN_BLOCK * IPT;
  static_assert(IPT % VEC == 0, "items per thread must be whole vectors");

  __shared__ unsigned s_tile;
  using prefix_smem_t = tile_prefix_smem<T, NWARPS>;
  TB200_SHARED_OBJECT(prefix_smem_t, sm);

  if (one_cluster) {
    if (threadIdx.x == 0) s_tile = blockIdx.x;
    if (blockIdx.x == 0 && threadIdx.x < sizeof(ws_header) / 4) reinterpret_cast<unsigned*>(hdr)[threadIdx.x] = 0;   // nobody has cleared it
  } else if (threadIdx.x == 0) s_tile = atomicAdd(&hdr->ticket, 1u);
  __syncthreads();
  const size_t tile = s_tile;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const size_t wbase = tile * TILE + (size_t)warp * WCHUNK;
  const bool full = tile * TILE + TILE <= n;

  T x[VPT][VEC];
  // ---- load: vector v of this lane covers items wbase + (v*32 + lane)*VEC ... +VEC
  if constexpr (VEC > 1) {
    if (full) {
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        vec16 r = load_stream16(reinterpret_cast<const char*>(in) + (wbase + (size_t)(v * 32 + lane) * VEC) * sizeof(T));
        const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
        for (int k = 0; k < VEC; ++k) x[v][k] = e[k];
      }
    } else {
#pragma unroll
      for (int v = 0; v < VPT; ++v)
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
          size_t i = wbase + (size_t)(v * 32 + lane) * VEC + k;
          x[v][k] = i < n ? (T)in[i] : T();
        }
    }
  } else {
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      size_t i = wbase + (size_t)(v * 32 + lane);
      if (full || i < n) x[v][0] = (T)in[i]; else x[v][0] = T();
    }
  }

  // ---- scan inside each vector, then chain vector totals: warp rows, warps, preceding tiles
  T vec_total[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
#pragma unroll
    for (int k = 1; k < VEC; ++k) x[v][k] = op(x[v][k - 1], x[v][k]);
    vec_total[v] = x[v][VEC - 1];
  }
  opt<T> pre[VPT];   // everything before vector v of this lane, across tiles, including init
  tile_exclusive_prefix<T, Op, VPT, NWARPS>(vec_total, pre, tile, init, has_init, op, ts, &rep->error, sm, one_cluster);

  // ---- apply and store
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const opt<T> E = pre[v];
    T y[VEC];
    if (INCLUSIVE) {
#pragma unroll
      for (int k = 0; k < VEC; ++k) y[k] = E.has ? op(E.v, x[v][k]) : x[v][k];
    } else {
      y[0] = E.v;
#pragma unroll
      for (int k = 1; k < VEC; ++k) y[k] = op(E.v, x[v][k - 1]);
    }
    const size_t i0 = wbase + (size_t)(v * 32 + lane) * VEC;
    if constexpr (VEC > 1) {
      if (full) {
        vec16 r;
        T* e = reinterpret_cast<T*>(&r);
#pragma unroll
        for (int k = 0; k < VEC; ++k) e[k] = y[k];
        store_stream16(reinterpret_cast<char*>(out) + i0 * sizeof(T), r);
      } else {
#pragma unroll
        for (int k = 0; k < VEC; ++k) if (i0 + k < n) out[i0 + k] = y[k];
      }
    } else {
      if (full || i0 < n) out[i0] = y[0];
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Windowed route, for inputs that the copy engine cannot fetch (any random-access iterator over a large
// range): reduce, fold, scan over one window of the input at a time, so that the second evaluation of the
// iterator finds its window in the 126 MB L2 and HBM sees every element once on the way in and once on the
// way out.  (transform_inclusive_scan of 2^28 int32: 0.54 ms, against 0.845 ms on the single-pass kernel.)
//
// One persistent kernel, one CTA per resident slot (`gridDim.x` CTAs, all resident: the host sizes the
// grid from the occupancy query).  Window w is the tiles [w * G * TPC, (w + 1) * G * TPC); CTA c owns the
// chunk of TPC consecutive tiles number c in every window.  Per window a CTA
//   A: reduces its chunk (plain loads: the lines stay in L2) and publishes the total in a
//      descriptor (value and status in one word);
//   F: folds the descriptors of the whole window -- the totals of the chunks before its own give
//      its carry, all of them the running total for the next window; the wait for a descriptor is
//      bounded, and since A of window w + 1 is issued BEFORE F of window w, the other CTAs' totals
//      have normally arrived long before they are asked for;
//   B: scans its chunk front to back (evict-first loads that hit L2, streaming stores), the carry
//      passing from tile to tile in registers.
// Every CTA publishes A(w) before it waits for anything of window w, so the waits cannot deadlock
// as long as all CTAs are resident; CTAs are never more than one window apart, so about two windows
// of input and two of output are live in L2 at a time.
constexpr int SCANW_CTAS_PER_SM = 4;
template <class T> struct scanw_tuning { static constexpr int IPT = (int)(64 / sizeof(T)); };   // 64 bytes per thread and tile
constexpr size_t SCANW_MIN_TILES_PER_CTA = 2;   // shorter inputs take the single-pass kernel
constexpr size_t SCANW_MAX_GRID = 2048;   // CTAs at most (the fold gives every thread GRID / 256 descriptors)
#ifndef TB200_SCANW_TPC
#define TB200_SCANW_TPC 3        // tiles per chunk: window = resident CTAs * TPC * 16 KB (28 MB on a B200; 2 and 3 measured alike, 1 and 4+ slower)
#endif

template <class T, class Op> __device__ __forceinline__ T warp_reduce_id(T x, Op op) {
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) x = op(x, shfl_generic(x, 0, 3, d));   // butterfly: the operators here commute
  return x;
}

// InIt: any random-access iterator whose values convert to T, one element per load.
template <class InIt, class T, class Op, bool INCLUSIVE, int VEC, int IPT>
__global__ void __launch_bounds__(SCAN_BLOCK, SCANW_CTAS_PER_SM)
scan_window_kernel(InIt in, T* out, size_t n, size_t tiles, unsigned tiles_per_chunk, T init, bool has_init, const T* init_ptr, Op op,
                   tile_state<T> ts, ws_header* hdr) {
  if (init_ptr) { init = *init_ptr; has_init = true; }
  constexpr int VPT = IPT / VEC;
  constexpr int NWARPS = SCAN_BLOCK / 32;
  constexpr size_t WT = 32 * IPT;           // a warp's tile: each lane holds VPT 16-byte vectors, lane-interleaved
  const T ID = op_identity<Op, T>::value();
  __shared__ T s_part[2][NWARPS];          // each warp's total of its part of the chunk, by window parity
  __shared__ T s_fold[2][NWARPS];          // per warp: fold of the chunks before this CTA's, of all chunks
  __shared__ T s_first;                    // what a loop would start from (drops_nans)
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const size_t G = gridDim.x, c = blockIdx.x;
  const size_t wtiles = (n + WT - 1) / WT;
  const size_t chunk_wtiles = (size_t)tiles_per_chunk * NWARPS;   // a CTA's chunk; warp w owns the w-th run of tiles_per_chunk warp tiles
  const size_t windows = (wtiles + G * chunk_wtiles - 1) / (G * chunk_wtiles);
  (void)tiles;

  auto chunk_first = [&](size_t w, size_t chunk) { return (w * G + chunk) * chunk_wtiles; };
  auto load_tile = [&](vec16 (&r)[VPT], size_t wt) {
    const size_t base = wt * WT;
    const bool full = base + WT <= n;
    if (full) {
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        T* e = reinterpret_cast<T*>(&r[v]);
#pragma unroll
        for (int k = 0; k < VEC; ++k) e[k] = no_nan<Op>((T)in[base + (size_t)(v * 32 + lane) * VEC + k]);
      }
    } else {
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        T* e = reinterpret_cast<T*>(&r[v]);
#pragma unroll
        for (int k = 0; k < VEC; ++k) {
          const size_t i = base + (size_t)(v * 32 + lane) * VEC + k;
          e[k] = i < n ? no_nan<Op>((T)in[i]) : ID;
        }
      }
    }
  };
  // A: every warp reduces its part of the CTA's chunk of window w; the CTA's total is published
  auto phase_a = [&](size_t w) {
    const size_t first = chunk_first(w, c);
    if (first >= wtiles) return;
    const size_t mine = first + (size_t)warp * tiles_per_chunk;
    T acc = ID;
    for (unsigned t = 0; t < tiles_per_chunk; ++t) {
      if (mine + t >= wtiles) break;
      vec16 r[VPT];
      load_tile(r, mine + t);
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const T* e = reinterpret_cast<const T*>(&r[v]);
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc = op(acc, e[k]);
      }
    }
    acc = warp_reduce_id(acc, op);
    T* part = s_part[w & 1];
    if (lane == 0) part[warp] = acc;
    __syncthreads();
    if (warp == 0) {
      T t = lane < NWARPS ? part[lane] : ID;
      t = warp_reduce_id(t, op);
      if (lane == 0) ts.publish(w * G + c, TILE_AGGREGATE, t);
    }
  };

  T running = has_init ? no_nan<Op>(init) : ID;   // init (+) everything before the current window
  if constexpr (drops_nans<Op, T>::value) {
    // read before this CTA publishes, so before anybody stores: the iterator may read from where the output goes
    if (threadIdx.x == 0) s_first = has_init ? init : (T)in[0];
    __syncthreads();
  }
  phase_a(0);
  for (size_t w = 0; w < windows; ++w) {
    if (w + 1 < windows) phase_a(w + 1);
    const size_t first = chunk_first(w, c);
    if (first >= wtiles) break;   // only in the last window: no chunk of this CTA, and nobody waits for it
    // ---- F: fold the window's descriptors: every thread polls a few (all loads in flight at once),
    // each warp leaves its partial fold in shared memory
    {
      constexpr int SLOTS = (int)(SCANW_MAX_GRID / SCAN_BLOCK);
      T v[SLOTS];
      unsigned st[SLOTS];
#pragma unroll
      for (int j = 0; j < SLOTS; ++j) {
        const size_t k = threadIdx.x + (size_t)j * SCAN_BLOCK;
        st[j] = TILE_AGGREGATE; v[j] = ID;
        if (k < G && chunk_first(w, k) < wtiles) st[j] = ts.poll(w * G + k, v[j]);
      }
      T before = ID, total = ID;
#pragma unroll
      for (int j = 0; j < SLOTS; ++j) {
        const size_t k = threadIdx.x + (size_t)j * SCAN_BLOCK;
        unsigned iter = 0;
        while (st[j] == TILE_INVALID) {
          if (++iter > SPIN_LIMIT) { record_error(&hdr->error, ERR_LOOKBACK_TIMEOUT); v[j] = ID; break; }
          backoff(iter);
          st[j] = ts.poll(w * G + k, v[j]);
        }
        if (k < c) before = op(before, v[j]);
        total = op(total, v[j]);
      }
      before = warp_reduce_id(before, op);
      total = warp_reduce_id(total, op);
      if (lane == 0) { s_fold[0][warp] = before; s_fold[1][warp] = total; }
    }
    __syncthreads();
    // this warp's carry: init and the windows before, the chunks before this CTA's, the warps before this one
    T carry;
    {
      T before = ID, total = ID;
#pragma unroll
      for (int w2 = 0; w2 < NWARPS; ++w2) { before = op(before, s_fold[0][w2]); total = op(total, s_fold[1][w2]); }
      carry = op(running, before);
      running = op(running, total);
      const T* part = s_part[w & 1];
#pragma unroll
      for (int w2 = 0; w2 < NWARPS; ++w2) if (w2 < warp) carry = op(carry, part[w2]);
    }
    // ---- B: the warp scans its part of the chunk, tile after tile, no barrier
    const size_t mine = first + (size_t)warp * tiles_per_chunk;
    for (unsigned t = 0; t < tiles_per_chunk; ++t) {
      const size_t wt = mine + t;
      if (wt >= wtiles) break;
      vec16 r[VPT];
      load_tile(r, wt);
      T x[VPT][VEC];
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const T* e = reinterpret_cast<const T*>(&r[v]);
#pragma unroll
        for (int k = 0; k < VEC; ++k) x[v][k] = e[k];
      }
      T pre[VPT];   // carry (+) everything of this tile before vector v of this lane
      T rowacc = carry;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
#pragma unroll
        for (int k = 1; k < VEC; ++k) x[v][k] = op(x[v][k - 1], x[v][k]);
        const T incl = warp_inclusive_scan(x[v][VEC - 1], op);
        T lanepref = shfl_up(incl, 1);
        if (lane == 0) lanepref = ID;
        pre[v] = op(rowacc, lanepref);
        rowacc = op(rowacc, shfl_idx(incl, 31));
      }
      carry = rowacc;
      const size_t base = wt * WT;
      const bool full = base + WT <= n;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const T E = pre[v];
        T y[VEC];
        if (INCLUSIVE) {
#pragma unroll
          for (int k = 0; k < VEC; ++k) y[k] = op(E, x[v][k]);
        } else {
          y[0] = E;
#pragma unroll
          for (int k = 1; k < VEC; ++k) y[k] = op(E, x[v][k - 1]);
        }
        if constexpr (drops_nans<Op, T>::value) {
          const T first = s_first;
#pragma unroll
          for (int k = 0; k < VEC; ++k) if (first != first) y[k] = first;
        }
        const size_t i0 = base + (size_t)(v * 32 + lane) * VEC;
        if (full) {
          vec16 o;
          T* e = reinterpret_cast<T*>(&o);
#pragma unroll
          for (int k = 0; k < VEC; ++k) e[k] = y[k];
          store_stream16(reinterpret_cast<char*>(out) + i0 * sizeof(T), o);
        } else {
#pragma unroll
          for (int k = 0; k < VEC; ++k) if (i0 + k < n) out[i0 + k] = y[k];
        }
      }
    }
    __syncthreads();   // s_fold is rewritten in the next window
  }
}

// Resident CTAs of the windowed kernel on the current device (cached per kernel and device).
template <class Kernel> int resident_ctas(Kernel kernel, int block, size_t smem) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem) != cudaSuccess || per_sm < 1) return 0;
  return per_sm * current_device_info().sm_count;
}

// Where the pipeline starts (a call and the wait for it): 1 M int32 14.2 us against 16.2 single-pass, 2^19 13.7 against 13.9, 400 k
// 13.9 against 13.6.
constexpr size_t SCAN_PIPE_MIN_BYTES = (size_t)1 << 21;
// inputs of two tiles and more for every CTA of the windowed kernel: where that one starts
template <class T> bool scan_fills_windows(size_t n) {
  const size_t tile = (size_t)SCAN_BLOCK * scanw_tuning<T>::IPT, ctas = (size_t)current_device_info().sm_count * SCANW_CTAS_PER_SM;
  return (n + tile - 1) / tile >= SCANW_MIN_TILES_PER_CTA * ctas;
}

template <class T> size_t scan_tile_items() { return (size_t)SCAN_BLOCK * scan_tuning<T>::IPT; }
// descriptors of the windowed route: one per chunk, the last window padded to a whole grid
template <class T> size_t scanw_descriptor_bound(size_t n) {
  const size_t tile = (size_t)SCAN_BLOCK * scanw_tuning<T>::IPT;
  return ((n + tile - 1) / tile + TB200_SCANW_TPC - 1) / TB200_SCANW_TPC + SCANW_MAX_GRID;
}
template <class T> size_t scan_workspace_bytes(size_t n) {   // every route fits
  size_t tiles = (n + scan_tile_items<T>() - 1) / scan_tile_items<T>();
  size_t need = tile_state<T>::bytes(tiles + 1);   // single pass
  if (tile_state_mode<T>::value != 0 && tile_state<T>::bytes(scanw_descriptor_bound<T>(n)) > need) need = tile_state<T>::bytes(scanw_descriptor_bound<T>(n));
  if constexpr (std::is_arithmetic<T>::value && (sizeof(T) == 4 || sizeof(T) == 8)) {
    const size_t pipe = scan_pipe_descriptor_bytes<T>(n);
    if (pipe > need) need = pipe;
  }
  return sizeof(ws_header) + need;
}

// The windowed route: launches it if the input is large enough for windows to pay (launched = true).
template <bool INCLUSIVE, class InIt, class T, class Op>
cudaError_t scan_window_launch(InIt in, T* out, size_t n, T init, bool has_init, const T* d_init, Op op, char* base, ws_header* hdr,
                               cudaStream_t stream, bool& launched) {
  launched = false;
  constexpr int VEC = 16 / sizeof(T);
  constexpr int IPT2 = scanw_tuning<T>::IPT;
  const size_t tiles2 = (n + (size_t)SCAN_BLOCK * IPT2 - 1) / ((size_t)SCAN_BLOCK * IPT2);
  auto kern = scan_window_kernel<InIt, T, Op, INCLUSIVE, VEC, IPT2>;
  static thread_local int resident[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && resident[dev] == 0) resident[dev] = resident_ctas(kern, SCAN_BLOCK, 0);
  size_t grid = (dev >= 0 && dev < 64) ? (size_t)resident[dev] : 0;
  if (grid > SCANW_MAX_GRID) grid = SCANW_MAX_GRID;
  const unsigned tpc = TB200_SCANW_TPC;
  if (grid == 0 || tiles2 < 2 * grid * tpc) return cudaSuccess;
  const size_t windows = (tiles2 + grid * tpc - 1) / (grid * tpc);
  tile_state<T> tsw;
  tsw.bind(base + sizeof(ws_header), windows * grid);
  cudaError_t e3 = cudaMemsetAsync(base, 0, sizeof(ws_header) + tile_state<T>::bytes(windows * grid), stream);
  if (e3 != cudaSuccess) return e3;
  launched = true;
  timed_launch tl(KID_SCAN, stream);
  kern<<<(unsigned)grid, SCAN_BLOCK, 0, stream>>>(in, out, n, tiles2, tpc, init, has_init, d_init, op, tsw, hdr);
  log_launch("scan_window_kernel", grid, SCAN_BLOCK, 0, n, stream);
  return cudaGetLastError();
}

// Launches the scan on `stream`; no sync.  in == out is allowed.  d_init, if not null, points at an
// initial value in device memory that replaces (init, has_init); it is read when the kernels run.
template <bool INCLUSIVE, class InIt, class OutIt, class T, class Op>
cudaError_t scan_async(InIt in, OutIt out, size_t n, T init, bool has_init, Op op, void* ws, cudaStream_t stream, const T* d_init = nullptr) {
  if (n == 0) return cudaMemsetAsync(ws, 0, sizeof(ws_header), stream);
  constexpr int IPT = scan_tuning<T>::IPT;
  const size_t tiles = (n + scan_tile_items<T>() - 1) / scan_tile_items<T>();
  char* base = static_cast<char*>(ws);
  ws_header* hdr = reinterpret_cast<ws_header*>(base);
  constexpr bool ptrs = std::is_pointer<InIt>::value && std::is_pointer<OutIt>::value;
  bool vectors = false;
  if constexpr (ptrs) {
    using In = typename std::remove_cv<typename std::remove_pointer<InIt>::type>::type;
    using Out = typename std::remove_pointer<OutIt>::type;
    constexpr bool vec_ok = std::is_same<In, T>::value && std::is_same<Out, T>::value && std::is_arithmetic<T>::value &&
                            (sizeof(T) == 4 || sizeof(T) == 8);
    if constexpr (vec_ok) {
      vectors = is_aligned16(in) && is_aligned16(out);
      if constexpr (is_commutative_op<Op>::value) {
        // With NaNs among the values the single-pass kernel's floating min and max depend on its grouping; the pipeline's
        // do not (drops_nans).  So that no size's results change with it, they leave the single-pass kernel where they always did.
        constexpr bool grouping_shows = drops_nans<Op, T>::value;
        if (vectors && (grouping_shows ? scan_fills_windows<T>(n) : n * sizeof(T) >= SCAN_PIPE_MIN_BYTES)) {
          bool launched = false;
          cudaError_t e2 = scan_pipe_launch<INCLUSIVE, T, Op>(in, out, n, init, has_init, d_init, ws, stream, launched);
          if (launched || e2 != cudaSuccess) return e2;
        }
      }
    }
  }
  // any other input iterator with a contiguous, aligned output of T: the windowed kernel with one
  // element per load (transform_inclusive_scan / transform_exclusive_scan over a device range)
  if constexpr (!std::is_pointer<InIt>::value && std::is_pointer<OutIt>::value && is_commutative_op<Op>::value) {
    using Out = typename std::remove_pointer<OutIt>::type;
    if constexpr (std::is_same<Out, T>::value && std::is_arithmetic<T>::value && (sizeof(T) == 4 || sizeof(T) == 8)) {
      if (is_aligned16(out) && scan_fills_windows<T>(n)) {
        bool launched = false;
        cudaError_t e3 = scan_window_launch<INCLUSIVE>(in, out, n, init, has_init, d_init, op, base, hdr, stream, launched);
        if (launched || e3 != cudaSuccess) return e3;
      }
    }
  }
  tile_state<T> ts;
  ts.bind(base + sizeof(ws_header), tiles + 1);
  ws_header* const rep = report_of(hdr, stream);
  auto launch = [&](auto vec_tag) -> cudaError_t {
    constexpr int VEC = decltype(vec_tag)::value;
    auto kern = scan_kernel<InIt, OutIt, T, Op, INCLUSIVE, VEC, IPT>;
    const char* const name = VEC > 1 ? "scan_kernel (16-byte loads)" : "scan_kernel (generic iterator)";
    timed_launch tl(KID_SCAN, stream);
    const unsigned ctas = cluster_ctas(tiles);
    if (cluster_storable<T>::value && ctas != 0 && !tiles_stay_apart()) {
      static thread_local unsigned largest[64] = {0};
      bool launched = false;
      const cudaError_t e = cluster_launch(kern, ctas, SCAN_BLOCK, 0, stream, largest, launched, in, out, n, init, has_init, d_init, op, ts, hdr, rep, true);
      if (launched) { reported(e, rep, hdr); log_launch(name, ctas, SCAN_BLOCK, 0, n, stream); }
      if (launched || e != cudaSuccess) return e;
    }
    cudaError_t e = cudaMemsetAsync(base, 0, sizeof(ws_header) + tile_state<T>::bytes(tiles + 1), stream);
    if (e != cudaSuccess) return e;
#ifdef TB200_TEST_HOOKS
    if (test_hook_flags() & 1u) { if ((e = cudaMemsetAsync(&hdr->flags, 1, 1, stream)) != cudaSuccess) return e; }
#endif
    kern<<<(unsigned)tiles, SCAN_BLOCK, 0, stream>>>(in, out, n, init, has_init, d_init, op, ts, hdr, rep, false);
    log_launch(name, tiles, SCAN_BLOCK, 0, n, stream);
    return reported(cudaGetLastError(), rep, hdr);
  };
  if constexpr (ptrs) {
    using In = typename std::remove_cv<typename std::remove_pointer<InIt>::type>::type;
    using Out = typename std::remove_pointer<OutIt>::type;
    constexpr bool vec_ok = std::is_same<In, T>::value && std::is_same<Out, T>::value && std::is_arithmetic<T>::value &&
                            (sizeof(T) == 4 || sizeof(T) == 8);
    if constexpr (vec_ok) {
      if (vectors) return launch(std::integral_constant<int, 16 / sizeof(T)>());
    }
  }
  return launch(std::integral_constant<int, 1>());
}

}  // namespace tb200
