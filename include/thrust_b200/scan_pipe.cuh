// Inclusive / exclusive scan of large contiguous inputs on sm_100a on the tile pipeline (tile_pipe.cuh), for
// operators with an identity on 4- and 8-byte arithmetic types (floating min and max without their NaNs, drops_nans).  A tile is read from HBM once into shared
// memory; the compute warps reduce it there ahead of time, and once its carry is known scan it from the
// same shared memory and stream the result out: 2 * sizeof(T) bytes of HBM traffic per element and no
// second trip of the input through L2.  Bound by HBM: 2^28 int32 or fp32 0.33 ms (6470 GB/s; 0.43 with the input
// read a second time out of L2, 0.62 in a single pass with look-back), 2^27 doubles 0.34 ms (0.54 single-pass).
#pragma once
#include "tile_pipe.cuh"

namespace tb200 {

template <class T, class Op, bool INCLUSIVE>
__global__ void __launch_bounds__(PIPE_BLOCK, 1)
scan_pipe_kernel(const T* in, T* out, size_t n, unsigned tiles, T init, bool has_init, const T* init_ptr, tile_chain<T, Op> chain, ws_header* rep) {
  using Chain = tile_chain<T, Op>;
  using C = typename Chain::C;
  constexpr int VEC = 16 / sizeof(T);
  constexpr int ITEMS = PIPE_TILE_BYTES / sizeof(T);
  extern __shared__ __align__(128) unsigned char pipe_raw[];
  __shared__ pipe_state<T, C> st;
  unsigned char* const stages = pipe_align(pipe_raw);
  const T ID = op_identity<Op, T>::value();
  const Op op = Op();
  pipe_init(st);
  const int lane = lane_id(), warp = threadIdx.x >> 5;

  if (warp == PIPE_LOADER) {
    const unsigned long long policy = l2_stream_policy();
    pipe_loader(st, tiles, &rep->error, [&](unsigned s, unsigned tile) {
      T* dst = reinterpret_cast<T*>(stages + (size_t)s * PIPE_TILE_BYTES);
      const size_t base = (size_t)tile * ITEMS;
      const unsigned bytes = pipe_tail_fill<T, ITEMS>(dst, in + base, n - base, ID);
      if (lane == 0) {
        mbar_arrive_expect(&st.full[s], bytes);
        if (bytes) bulk_load(dst, in + base, bytes, &st.full[s], policy);
      }
    });
  } else if (warp == PIPE_PUBLISHER) {
    pipe_publisher<false>(st, chain, tiles, &rep->error, [&](const T& part) {
      C t = lane < PIPE_WARPS ? Chain::lift(part) : Chain::identity();
#pragma unroll
      for (int d = 1; d < PIPE_WARPS; d <<= 1) t = Chain::join(t, shfl_down(t, d));   // lane 0: all parts, in order
      return t;
    });
  } else if (warp == PIPE_FOLDER) {
    C first = Chain::identity();
    if (init_ptr) first = Chain::lift(no_nan<Op>(*init_ptr)); else if (has_init) first = Chain::lift(no_nan<Op>(init));
    pipe_folder<false>(st, chain, tiles, first, &rep->error, [](const C&) {});
  } else {
    const int mine = warp % PIPE_WARPS;
    // what a loop would start from: if that is a NaN, so is every result (in place in[0] is stored unchanged)
    T first = T();
    if constexpr (drops_nans<Op, T>::value) first = init_ptr ? *init_ptr : has_init ? init : in[0];
    const bool stuck = first != first;
    auto rows_of = [&](unsigned s) { return reinterpret_cast<const vec16*>(stages + (size_t)s * PIPE_TILE_BYTES) + mine * (PIPE_ROWS * 32) + lane; };
    pipe_compute<false>(st, tiles, &rep->error,
      [&](unsigned s, unsigned) {
        const vec16* src = rows_of(s);
        T acc[PIPE_ROWS];
#pragma unroll
        for (int v = 0; v < PIPE_ROWS; ++v) {
          const vec16 r = src[v * 32];
          const T* e = reinterpret_cast<const T*>(&r);
          acc[v] = no_nan<Op>(e[0]);
#pragma unroll
          for (int k = 1; k < VEC; ++k) acc[v] = op(acc[v], no_nan<Op>(e[k]));
        }
#pragma unroll
        for (int v = 1; v < PIPE_ROWS; ++v) acc[0] = op(acc[0], acc[v]);
        T a = acc[0];
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) a = op(a, shfl_generic(a, 0, 3, d));   // butterfly: the operators here commute
        return a;
      },
      [&](unsigned s, unsigned tile) {
        const vec16* src = rows_of(s);
        T x[PIPE_ROWS][VEC];
#pragma unroll
        for (int v = 0; v < PIPE_ROWS; ++v) {
          const vec16 r = src[v * 32];
          const T* e = reinterpret_cast<const T*>(&r);
#pragma unroll
          for (int k = 0; k < VEC; ++k) x[v][k] = no_nan<Op>(e[k]);
        }
        // what precedes this warp's part: the tile's carry and the warps before this one
        T before = lane < mine ? st.part[s][lane & (PIPE_WARPS - 1)] : ID;
#pragma unroll
        for (int d = 1; d < PIPE_WARPS; d <<= 1) before = op(before, shfl_generic(before, 0, 3, d));
        const T carry = Chain::lower(Chain::join(st.carry[s], Chain::lift(shfl_idx(before, 0))));
        T pre[PIPE_ROWS];   // everything of this warp's part before vector v of this lane
        T rowacc = ID;
#pragma unroll
        for (int v = 0; v < PIPE_ROWS; ++v) {
#pragma unroll
          for (int k = 1; k < VEC; ++k) x[v][k] = op(x[v][k - 1], x[v][k]);
          const T incl = warp_inclusive_scan(x[v][VEC - 1], op);
          T lanepref = shfl_up(incl, 1);
          if (lane == 0) lanepref = ID;
          pre[v] = op(rowacc, lanepref);
          rowacc = op(rowacc, shfl_idx(incl, 31));
        }
        const size_t base = (size_t)tile * ITEMS + (size_t)mine * (PIPE_ROWS * 32 * VEC);
        const bool full = (size_t)tile * ITEMS + ITEMS <= n;
#pragma unroll
        for (int v = 0; v < PIPE_ROWS; ++v) {
          // floats: the part's own prefix first, so that only the last addition rounds at the carry's magnitude
          constexpr bool LATE = std::is_floating_point<T>::value;
          const T E = LATE ? pre[v] : op(carry, pre[v]);
          T y[VEC];
          if (INCLUSIVE) {
#pragma unroll
            for (int k = 0; k < VEC; ++k) y[k] = op(E, x[v][k]);
          } else {
            y[0] = E;
#pragma unroll
            for (int k = 1; k < VEC; ++k) y[k] = op(E, x[v][k - 1]);
          }
          if (LATE) {
#pragma unroll
            for (int k = 0; k < VEC; ++k) y[k] = op(carry, y[k]);
          }
          if constexpr (drops_nans<Op, T>::value) {
#pragma unroll
            for (int k = 0; k < VEC; ++k) if (stuck) y[k] = first;
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
      });
  }
}

template <class T> constexpr size_t scan_pipe_tile_items() { return PIPE_TILE_BYTES / sizeof(T); }
template <class T> size_t scan_pipe_descriptor_bytes(size_t n) {   // of the operator that needs most
  const size_t tiles = (n + scan_pipe_tile_items<T>() - 1) / scan_pipe_tile_items<T>();
  const size_t sum = tile_chain<T, plus_op>::bytes(tiles), other = tile_chain<T, min_op>::bytes(tiles);
  return sum > other ? sum : other;
}

// Launches the pipeline scan if the device can hold it and takes the launch (launched = true).  `in` and `out` are 16-byte aligned;
// they may be the same array.  The workspace holds the header and one descriptor per tile.
template <bool INCLUSIVE, class T, class Op>
cudaError_t scan_pipe_launch(const T* in, T* out, size_t n, T init, bool has_init, const T* d_init, void* ws, cudaStream_t stream, bool& launched) {
  launched = false;
  const size_t tiles = (n + scan_pipe_tile_items<T>() - 1) / scan_pipe_tile_items<T>();
  if (tiles >= 0xffffff00ull) return cudaSuccess;
  static thread_local bool ready[64] = {false};
  auto kern = scan_pipe_kernel<T, Op, INCLUSIVE>;
  const size_t smem = pipe_smem_bytes(PIPE_TILE_BYTES, 0);
  const size_t grid = pipe_grid(kern, smem, tiles, ready);
  if (grid == 0) return cudaSuccess;
  char* base = static_cast<char*>(ws);
  ws_header* hdr = reinterpret_cast<ws_header*>(base);
  tile_chain<T, Op> chain;
  chain.bind(base + sizeof(ws_header), tiles);
  cudaError_t e = pipe_clear(base, sizeof(ws_header) + tile_chain<T, Op>::bytes(tiles), stream);
  if (e != cudaSuccess) return e;
  timed_launch tl(KID_SCAN, stream);
  ws_header* const rep = report_of(hdr, stream);
  e = pipe_launch(kern, grid, smem, stream, in, out, n, (unsigned)tiles, init, has_init, d_init, chain, rep);
  if (launch_refused(e)) return cudaSuccess;
  reported(e, rep, hdr);
  launched = true;
  log_launch("scan_pipe_kernel", grid, PIPE_BLOCK, smem, n, stream);
  return e;
}

}  // namespace tb200
