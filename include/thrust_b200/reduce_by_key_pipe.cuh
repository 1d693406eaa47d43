// reduce_by_key of large contiguous inputs on sm_100a on the tile pipeline (tile_pipe.cuh), for 4- and
// 8-byte arithmetic keys and values (of one size or mixed) and operators with an identity.
//
// A tile, or a warp's part of it, is summarised by the pair
//     (number of run heads, reduction of the values behind its last head -- of all of them without a head),
// pairs combine as (c1, v1) (+) (c2, v2) = (c1 + c2, c2 ? v2 : op(v1, v2)), and a tile's descriptor is one
// 128-bit word: the value, and the count shifted over the status.  The compute warps summarise some tiles
// ahead; once a tile's carry is known they walk their items again (from shared memory) and emit, at every
// head, the head's key and the finished total of the run before it, compacted in place in shared
// memory and stored in 16-byte pieces.  The folder closes the last run.  Keys and values are read from HBM
// once.  fp32 sums are carried from tile to tile as doubles.
//
// Measured on B200, runs of mean length 4, against two streaming passes / one pass with look-back: 2^28 u32 + f32
// 0.71 ms (0.97 / 1.38), 2^27 u64 + f64 0.77 (0.95 / 2.15), 2^27 u32 + f64 0.71 (1.70 single-pass), 5 M u32 + f32 32 us
// (41).  Bound by the warps' instruction chains (segmented scan, compaction); the same bytes copied take 0.41 ms.
#pragma once
#include "tile_pipe.cuh"

namespace tb200 {

constexpr int RBK_PIPE_ROWS = 4;
template <class K, class V> struct rbk_pipe_shape {
  static constexpr int VEC = 16 / (int)(sizeof(K) > sizeof(V) ? sizeof(K) : sizeof(V));   // items per lane and row
  static constexpr int PART = RBK_PIPE_ROWS * 32 * VEC;                                   // items per compute warp and tile
  static constexpr int ITEMS = PIPE_WARPS * PART;
  using Keys = pipe_parts<K, PART>;
  using Vals = pipe_parts<V, PART>;
  static constexpr size_t STAGE_BYTES = Keys::BYTES + Vals::BYTES;
};

template <class V> struct rbk_part { unsigned heads; V value; };

template <class V, class Op> struct rbk_chain {
  // sums of fp32 values are carried in 64 bits
  using Wide = typename std::conditional<std::is_same<V, float>::value && std::is_same<Op, plus_op>::value, double, V>::type;
  struct C { unsigned long long heads; Wide value; };
  using R = C;
  unsigned long long* words;
  static size_t bytes(size_t tiles) { return align_up(tiles * 16, 256); }
  void bind(void* p, size_t) { words = static_cast<unsigned long long*>(p); }
  __device__ static C identity() { return C{0, (Wide)op_identity<Op, V>::value()}; }
  __device__ static C lift(const rbk_part<V>& p) { return C{p.heads, (Wide)p.value}; }
  __device__ static C join(const C& older, const C& newer) {
    C r;
    r.heads = older.heads + newer.heads;
    r.value = newer.heads ? newer.value : Op()(older.value, newer.value);
    return r;
  }
  __device__ static R start(const C& x) { return x; }
  __device__ static R extend(const R& r, const C& x) { return join(r, x); }
  __device__ static C value(const R& r) { return r; }
  // the first `count` descriptors of a round, descriptor j * 32 + lane in v[j]: all heads count, and of the values
  // those from the last descriptor with a head on
  __device__ static C fold_round(const C (&v)[PIPE_SLOTS], int count) {
    int from = 0;
#pragma unroll
    for (int j = 0; j < PIPE_SLOTS; ++j) {
      const unsigned heads = __ballot_sync(FULL_MASK, j * 32 + lane_id() < count && v[j].heads != 0);
      if (heads) from = j * 32 + 31 - __clz((int)heads);
    }
    C r = identity();
#pragma unroll
    for (int j = 0; j < PIPE_SLOTS; ++j) {
      if (j * 32 + lane_id() < count) {
        r.heads += v[j].heads;
        if (j * 32 + lane_id() >= from) r.value = Op()(r.value, v[j].value);
      }
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      r.heads += __shfl_xor_sync(FULL_MASK, r.heads, d);
      r.value = Op()(r.value, shfl_generic(r.value, 0, 3, d));
    }
    return r;
  }
  __device__ void publish(size_t tile, unsigned status, const C& v) const {
    unsigned long long bits = 0;
    memcpy(&bits, &v.value, sizeof(Wide));
    st_relaxed_b128(words + 2 * tile, bits, (v.heads << 2) | status);
  }
  __device__ unsigned poll(size_t tile, C& v) const {
    unsigned long long bits, w;
    ld_relaxed_b128(words + 2 * tile, bits, w);
    memcpy(&v.value, &bits, sizeof(Wide));
    v.heads = w >> 2;
    return (unsigned)w & 3u;
  }
};

// N consecutive items of a lane out of shared memory (8 or 16 bytes) into registers
template <class T, int N> __device__ __forceinline__ void lane_items(const T* p, T (&x)[N]) {
  static_assert(sizeof(T) * N == 16 || sizeof(T) * N == 8, "one vector load");
  if constexpr (sizeof(T) * N == 16) { const vec16 r = *reinterpret_cast<const vec16*>(p); memcpy(x, &r, 16); }
  else { const uint2 r = *reinterpret_cast<const uint2*>(p); memcpy(x, &r, 8); }
}

template <class K, class V, class Eq, class Op>
__global__ void __launch_bounds__(PIPE_BLOCK, 1)
rbk_pipe_kernel(const K* keys, const V* vals, K* keys_out, V* vals_out, size_t n, unsigned tiles, Eq eq, rbk_chain<V, Op> chain, ws_header* hdr,
                ws_header* rep, unsigned long long* d_count) {
  using Chain = rbk_chain<V, Op>;
  using C = typename Chain::C;
  using Shape = rbk_pipe_shape<K, V>;
  constexpr int VEC = Shape::VEC, PART = Shape::PART, ITEMS = Shape::ITEMS, ROWS = RBK_PIPE_ROWS;
  extern __shared__ __align__(128) unsigned char pipe_raw[];
  __shared__ pipe_state<rbk_part<V>, C> st;
  __shared__ __align__(16) vec16 s_edge[PIPE_STAGES];   // the keys in front of the stage's tile
  unsigned char* const stages = pipe_align(pipe_raw);
  const V ID = op_identity<Op, V>::value();
  const Op op = Op();
  pipe_init(st);
  const int lane = lane_id(), warp = threadIdx.x >> 5;

  // the fold of the parts held by lanes 0 ... PIPE_WARPS - 1, in order; result in lane 0
  auto fold_parts = [&](C t) {
#pragma unroll
    for (int d = 1; d < PIPE_WARPS; d <<= 1) t = Chain::join(t, shfl_down(t, d));
    return t;
  };

  if (warp == PIPE_LOADER) {
    const unsigned long long policy = l2_stream_policy();
    pipe_loader(st, tiles, &rep->error, [&](unsigned s, unsigned tile) {
      unsigned char* const kstage = stages + s * Shape::STAGE_BYTES;
      unsigned char* const vstage = kstage + Shape::Keys::BYTES;
      const size_t base = (size_t)tile * ITEMS, left = n - base;
      Shape::Keys::ragged(kstage, keys + base, left);
      Shape::Vals::ragged(vstage, vals + base, left);
      __syncwarp();
      if (lane == 0) {
        const unsigned front = tile > 0 ? 16u : 0u;
        mbar_arrive_expect(&st.full[s], Shape::Keys::bytes(left) + Shape::Vals::bytes(left) + front);
        if (front) bulk_load(&s_edge[s], keys + base - 16 / sizeof(K), front, &st.full[s], policy);
      }
      __syncwarp();
      if (lane < PIPE_WARPS) Shape::Keys::copy(kstage, keys + base, left, lane, &st.full[s], policy);
      else if (lane < 2 * PIPE_WARPS) Shape::Vals::copy(vstage, vals + base, left, lane - PIPE_WARPS, &st.full[s], policy);
    });
  } else if (warp == PIPE_PUBLISHER) {
    pipe_publisher<false>(st, chain, tiles, &rep->error, [&](const rbk_part<V>& part) { return fold_parts(lane < PIPE_WARPS ? Chain::lift(part) : Chain::identity()); });
  } else if (warp == PIPE_FOLDER) {
    pipe_folder<false>(st, chain, tiles, Chain::identity(), &rep->error, [&](const C& all) {
      vals_out[all.heads - 1] = (V)all.value;   // the last run ends with the input
      hdr->count = rep->count = all.heads;
      if (d_count) *d_count = all.heads;
    });
  } else {
    const int mine = warp % PIPE_WARPS;
    // the key in front of the stage's tile, for its first warp; the input's first key is compared with itself (and opens a
    // run whatever comes out), because `eq` may only ever see keys of the input
    auto tile_front = [&](unsigned s, unsigned tile) {
      return tile > 0 ? reinterpret_cast<const K*>(&s_edge[s])[16 / sizeof(K) - 1] : Shape::Keys::part(stages + s * Shape::STAGE_BYTES, 0)[0];
    };
    // this lane's items, and their head flags (bit v * VEC + k, held from a tile's summary to its end: 2^27 u32 + f32 352 us, 368 with the
    // flags found twice); items past the end are no heads and hold the identity; `edge`: the key in front of the warp's part
    open_words head_words;
    auto load_items = [&](unsigned s, K (&k)[ROWS][VEC], V (&x)[ROWS][VEC]) {
      const K* kp = Shape::Keys::part(stages + s * Shape::STAGE_BYTES, mine);
      const V* vp = Shape::Vals::part(stages + s * Shape::STAGE_BYTES + Shape::Keys::BYTES, mine);
#pragma unroll
      for (int v = 0; v < ROWS; ++v) {
        lane_items<K, VEC>(kp + (v * 32 + lane) * VEC, k[v]);
        lane_items<V, VEC>(vp + (v * 32 + lane) * VEC, x[v]);
      }
    };
    // items past the end hold the identity
    auto blank_past_end = [&](unsigned tile, V (&x)[ROWS][VEC]) {
      const size_t first = (size_t)tile * ITEMS + (size_t)mine * PART;
      if (first + PART <= n) return;
#pragma unroll
      for (int v = 0; v < ROWS; ++v) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) if (first + (size_t)(v * 32 + lane) * VEC + j >= n) x[v][j] = ID;
      }
    };
    auto heads_of = [&](unsigned tile, const K& edge, const K (&k)[ROWS][VEC]) {
      const size_t first = (size_t)tile * ITEMS + (size_t)mine * PART;
      unsigned bits = 0;
      auto scan_heads = [&](auto whole_tag) {
        constexpr bool WHOLE = decltype(whole_tag)::value;   // no item past the end
#pragma unroll
        for (int v = 0; v < ROWS; ++v) {
          K prev = shfl_up(k[v][VEC - 1], 1);
          const K wrap = v > 0 ? shfl_idx(k[v > 0 ? v - 1 : 0][VEC - 1], 31) : edge;
          if (lane == 0) prev = wrap;
#pragma unroll
          for (int j = 0; j < VEC; ++j) {
            const bool in = WHOLE || first + (size_t)(v * 32 + lane) * VEC + j < n;
            if (in && !eq(j == 0 ? prev : k[v][j > 0 ? j - 1 : 0], k[v][j])) bits |= 1u << (v * VEC + j);
          }
        }
      };
      if (first + PART <= n) scan_heads(std::true_type()); else scan_heads(std::false_type());
      if (first == 0 && lane == 0) bits |= 1u;   // the input's first item opens a run
      return bits;
    };
    constexpr unsigned ROW_BITS = (1u << VEC) - 1;
    // reduction of a lane's items of a row behind its last head there (of all of them without a head)
    auto tail_of = [&](unsigned row_bits, const V (&x)[VEC]) {
      V t = x[0];
#pragma unroll
      for (int j = 1; j < VEC; ++j) t = (row_bits >> j) & 1 ? x[j] : op(t, x[j]);
      return t;
    };
    pipe_compute<true>(st, tiles, &rep->error,
      [&](unsigned s, unsigned tile) {
        K k[ROWS][VEC]; V x[ROWS][VEC];
        // nobody compacts its part of this tile before every warp has been here
        unsigned char* const kstage = stages + s * Shape::STAGE_BYTES;
        const K edge = mine > 0 ? Shape::Keys::part(kstage, mine > 0 ? mine - 1 : 0)[PART - 1] : tile_front(s, tile);
        load_items(s, k, x);
        blank_past_end(tile, x);
        const unsigned bits = heads_of(tile, edge, k);
        head_words.put(bits);
        // only what lies behind the part's last head counts: later rows entirely, the head's row from the head's lane on
        V open = ID;
        bool live = true;   // no head behind the current row
#pragma unroll
        for (int v = ROWS - 1; v >= 0; --v) {
          const unsigned row = (bits >> (v * VEC)) & ROW_BITS;
          const unsigned heads = __ballot_sync(FULL_MASK, row != 0);
          const int from = heads ? 31 - __clz((int)heads) : 0;
          if (live && lane >= from) open = op(tail_of(row, x[v]), open);
          live = live && heads == 0;
        }
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const V y = shfl_down(open, d); open = op(open, y); }   // lane 0 (others run past the end harmlessly)
        rbk_part<V> p;
        p.heads = __reduce_add_sync(FULL_MASK, (unsigned)__popc(bits));
        p.value = open;
        return p;
      },
      [&](unsigned s, unsigned tile) {
        K k[ROWS][VEC]; V x[ROWS][VEC];
        load_items(s, k, x);
        blank_past_end(tile, x);
        const unsigned bits = head_words.take();
        K* const kbuf = Shape::Keys::part(stages + s * Shape::STAGE_BYTES, mine);
        V* const vbuf = Shape::Vals::part(stages + s * Shape::STAGE_BYTES + Shape::Keys::BYTES, mine);
        __syncwarp();   // every lane has its items: the parts may be overwritten
        C carry = fold_parts(lane < mine ? Chain::lift(st.part[s][lane & (PIPE_WARPS - 1)]) : Chain::identity());   // the warps before this one
        carry = Chain::join(st.carry[s], shfl_idx(carry, 0));
        const unsigned long long run0 = carry.heads;    // runs begun in front of this warp's part
        V row_carry = (V)carry.value;                   // the open run's total so far
        // heads before this lane in each row: one scan over the lanes for all rows
        static_assert(ROWS <= 4 && 32 * VEC <= 255, "a row's count fits a byte");
        unsigned packed = 0;
#pragma unroll
        for (int v = 0; v < ROWS; ++v) packed |= (unsigned)__popc((bits >> (v * VEC)) & ROW_BITS) << (8 * v);
        const unsigned incl = warp_inclusive_scan(packed, plus_op());
        const unsigned totals = __shfl_sync(FULL_MASK, incl, 31);
        const unsigned excl = incl - packed;
        // What is stored lies inside the outputs, else it is reported and nothing is stored: the heads held are those of this stage and
        // the carry leaves room.  (A store cannot hit the input: rbk_pipe_eligible.)
        const unsigned part_heads = __reduce_add_sync(FULL_MASK, (unsigned)__popc(bits));
        if (part_heads != st.part[s][mine].heads || run0 > (size_t)tile * ITEMS + (size_t)mine * PART) {
          if (lane == 0) record_error(&rep->error, ERR_INCONSISTENT);
          return;
        }
        const unsigned kshift = run_shift(keys_out + run0);
        const unsigned vshift = run_shift(vals_out + run0 - 1);   // a value belongs to the run before its head
        unsigned row_off = 0;
#pragma unroll
        for (int v = 0; v < ROWS; ++v) {
          const unsigned row = (bits >> (v * VEC)) & ROW_BITS;
          const unsigned heads = __ballot_sync(FULL_MASK, row != 0);
          const unsigned upto = heads & (0xffffffffu >> (31 - lane));
          const int segment = upto ? 31 - __clz((int)upto) : 0;   // first lane of this lane's segment
          V t = tail_of(row, x[v]);
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) { const V y = shfl_up(t, d); if (lane - d >= segment) t = op(y, t); }
          const V before = shfl_up(t, 1);
          const bool from_start = (heads & ((1u << lane) - 1)) == 0;   // what precedes the row continues into this lane
          V acc = from_start ? (lane == 0 ? row_carry : op(row_carry, before)) : before;
          unsigned r = row_off + ((excl >> (8 * v)) & 255);
#pragma unroll
          for (int j = 0; j < VEC; ++j) {
            const bool head = (row >> j) & 1;
            if (head) { kbuf[kshift + r] = k[v][j]; vbuf[vshift + r] = acc; }
            acc = head ? x[v][j] : op(acc, x[v][j]);
            r += head;
          }
          const V open = shfl_idx(t, 31);
          row_carry = heads ? open : op(row_carry, open);
          row_off += (totals >> (8 * v)) & 255;
        }
        __syncwarp();
        warp_store_run(keys_out + run0 - kshift, kbuf, kshift, kshift + row_off);
        // the value staged first belongs to run run0 - 1; the input's first head closes nothing
        const unsigned skip = run0 == 0 ? 1u : 0u;
        if (row_off > skip) warp_store_run(vals_out + run0 - 1 - vshift, vbuf, vshift + skip, vshift + row_off);
      });
  }
}

// Whether the pipeline may serve a call: 16-byte aligned inputs that no output overlaps.
template <class K, class V>
bool rbk_pipe_eligible(const K* keys, const V* vals, const K* keys_out, const V* vals_out, size_t n) {
  if (!is_aligned16(keys) || !is_aligned16(vals)) return false;
  auto apart = [n](const void* in, size_t in_size, const void* out, size_t out_size) {
    const char* i = static_cast<const char*>(in);
    const char* o = static_cast<const char*>(out);
    return o >= i + n * in_size || i >= o + n * out_size;
  };
  return apart(keys, sizeof(K), keys_out, sizeof(K)) && apart(keys, sizeof(K), vals_out, sizeof(V)) && apart(vals, sizeof(V), keys_out, sizeof(K)) &&
         apart(vals, sizeof(V), vals_out, sizeof(V));
}

template <class K, class V> size_t rbk_pipe_workspace_bytes(size_t n) {
  return sizeof(ws_header) + rbk_chain<V, plus_op>::bytes((n + rbk_pipe_shape<K, V>::ITEMS - 1) / rbk_pipe_shape<K, V>::ITEMS);
}

// Launches the pipeline if the device can hold it and takes the launch (launched = true); n > 0.
template <class K, class V, class Eq, class Op>
cudaError_t rbk_pipe_launch(const K* keys, const V* vals, K* keys_out, V* vals_out, size_t n, Eq eq, unsigned long long* d_count, void* ws, cudaStream_t stream,
                            bool& launched) {
  launched = false;
  using Shape = rbk_pipe_shape<K, V>;
  const size_t tiles = (n + Shape::ITEMS - 1) / Shape::ITEMS;
  if (tiles >= 0xffffff00ull) return cudaSuccess;
  static thread_local bool ready[64] = {false};
  auto kern = rbk_pipe_kernel<K, V, Eq, Op>;
  const size_t smem = pipe_smem_bytes(Shape::STAGE_BYTES, 0);
  const size_t grid = pipe_grid(kern, smem, tiles, ready);
  if (grid == 0) return cudaSuccess;
  char* base = static_cast<char*>(ws);
  ws_header* hdr = reinterpret_cast<ws_header*>(base);
  rbk_chain<V, Op> chain;
  chain.bind(base + sizeof(ws_header), tiles);
  cudaError_t e = pipe_clear(base, sizeof(ws_header) + rbk_chain<V, Op>::bytes(tiles), stream);
  if (e != cudaSuccess) return e;
  timed_launch tl(KID_REDUCE_BY_KEY, stream);
  ws_header* const rep = report_of(hdr, stream);
  e = pipe_launch(kern, grid, smem, stream, keys, vals, keys_out, vals_out, n, (unsigned)tiles, eq, chain, hdr, rep, d_count);
  if (launch_refused(e)) return cudaSuccess;
  reported(e, rep, hdr);
  launched = true;
  log_launch("rbk_pipe_kernel", grid, PIPE_BLOCK, smem, n, stream);
  return e;
}

}  // namespace tb200
