// The tile pipeline shared by the streaming kernels for large inputs (scan, compaction, reduce_by_key)
// on sm_100a: every element is read from HBM once, by the copy engine, and a tile's prefix is known
// before the tile is needed.
//
// One persistent CTA per SM; CTA c owns the tiles c, c + G, c + 2G, ... of the input (G CTAs, launched
// cooperatively: all of them are resident).  A tile lives in one stage of a ring in shared memory from the moment
// it is loaded until its results are written.  Roles inside the CTA:
//   loader     (1 warp)   fills free stages with bulk copies (cp.async.bulk, completion on an mbarrier);
//   compute    (2 groups of 8 warps, tiles in turn) summarise tiles up to LOOKAHEAD ahead and finish the oldest
//                         one: both work in shared memory only, and a warp does whichever can be done.  A tile's way
//                         through a warp is a chain of shuffles and shared-memory trips, so what counts is how many
//                         rows a warp has in flight and how many tiles are worked on at a time;
//   publisher  (1 warp)   folds the warps' summaries of a tile and publishes the tile's descriptor (value
//                         and status in one word) for the other CTAs;
//   folder     (1 warp)   reads all G descriptors of its current round (round i: tiles iG ... iG + G - 1): those
//                         of the CTAs before it give the tile's carry, all of them the running total that the
//                         next round starts from.
// A round costs a CTA one coalesced read of the others' descriptors, and because tiles are summarised LOOKAHEAD
// tiles before they are finished, the descriptors are normally there.  Nothing waits in a circle: a tile's
// descriptor depends on its own load and on the carries of earlier rounds only.  Every wait is bounded; when one
// runs out the CTA records ERR_LOOKBACK_TIMEOUT, stops waiting and runs to its end.
//
// Why this shape.  At the copy rate of HBM an SM gets a 32 KB tile (read and written) every 2800 cycles, a few times
// the latency of a descriptor's way to the other CTAs; four tiles may be summarised and open while the next two
// load.  Measured on 2^28 int32 scanned: without any chaining 0.321 ms; this 0.332 ms (2 * 4 * n bytes at 6470 GB/s);
// 16 KB tiles 0.414; with tiles by an atomic ticket and a look-back to the nearest inclusive prefix instead of
// rounds 0.48 ms at best -- a tile's turn then waits for whole chains of look-backs.  One group of 16 warps, four rows
// each, instead of two of 8 does the scan as fast, but unique in 0.381 ms instead of 0.322 and reduce_by_key
// in 0.99 instead of 0.71; three tiles of a group open instead of two leave too few stages to load (unique 0.337).
#pragma once
#include "bulk_copy.cuh"
#include "common.cuh"

namespace tb200 {

constexpr int PIPE_WARPS = 8;                             // compute warps per group: a tile is one group's
constexpr int PIPE_GROUPS = 2;
constexpr int PIPE_LOADER = PIPE_GROUPS * PIPE_WARPS, PIPE_PUBLISHER = PIPE_LOADER + 1, PIPE_FOLDER = PIPE_LOADER + 2;   // warps
constexpr int PIPE_BLOCK = (PIPE_FOLDER + 1) * 32;
constexpr int PIPE_TILE_BYTES = 32768;
constexpr int PIPE_ROWS = PIPE_TILE_BYTES / 512 / PIPE_WARPS;   // 512-byte rows (32 lanes x 16 bytes) of a tile per compute warp
constexpr int PIPE_LOOKAHEAD = 1;                         // tiles of a group summarised ahead of the one being finished
constexpr int PIPE_STAGES = 6;
constexpr int PIPE_SLOTS = 5;                             // descriptors per lane of the folder
constexpr int PIPE_MAX_GRID = 32 * PIPE_SLOTS;            // CTAs at most (148 on a B200)
constexpr unsigned PIPE_POLL_NS = 100;                    // between two looks at descriptors that were not there

// ---------------------------------------------------------------- waiting
// Bounded wait for the phase of `bar` with the given parity.  `dead` (shared) is set once any wait of the
// CTA has run out; from then on nothing waits any more.
__device__ __forceinline__ void pipe_wait(unsigned long long* bar, unsigned parity, volatile unsigned* dead, unsigned* err) {
  unsigned iter = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (*dead) return;
    if (++iter > MBAR_SPIN_LIMIT) { *dead = 1; record_error(err, ERR_LOOKBACK_TIMEOUT); return; }
  }
}

// ---------------------------------------------------------------- operators with an identity
// The operators of this route have an identity, so nothing here needs the "value may be absent"
// bookkeeping of the generic kernels: plus starts from -0.0 for floating point (x + -0.0 == x for
// every x, signed zeros included) and 0 otherwise, min from the largest and max from the smallest value.
// Floating min and max take NaNs out first, see drops_nans.
template <class Op, class T> struct op_identity;
template <class T> struct op_identity<plus_op, T> {
  __host__ __device__ static T value() { return std::is_floating_point<T>::value ? (T)-0.0 : (T)0; }
};
template <class T> struct op_identity<min_op, T> {
  __host__ __device__ static T value() {
    if constexpr (std::is_floating_point<T>::value) return (T)INFINITY;
    else if constexpr (std::is_signed<T>::value) return (T)(((unsigned long long)1 << (8 * sizeof(T) - 1)) - 1);
    else return (T)~(T)0;
  }
};
template <class T> struct op_identity<max_op, T> {
  __host__ __device__ static T value() {
    if constexpr (std::is_floating_point<T>::value) return (T)-INFINITY;
    else if constexpr (std::is_signed<T>::value) return (T)((unsigned long long)1 << (8 * sizeof(T) - 1));
    else return (T)0;
  }
};

// Floating min and max one after the other, as a loop applies them: min_op(a, b) keeps a NaN that stands on its left
// and drops one on its right, so the result is the first value of all if that is a NaN, else the extreme of
// the values that are none.  With NaNs about the infinities are no identities and the grouping shows; so a scan replaces
// every NaN by the identity as it loads it (no_nan) and looks at the first value by itself.  Without NaNs nothing changes.
template <class Op, class T> struct drops_nans {
  static constexpr bool value = std::is_floating_point<T>::value && (std::is_same<Op, min_op>::value || std::is_same<Op, max_op>::value);
};
template <class Op, class T> __device__ __forceinline__ T no_nan(const T& x) {
  if constexpr (drops_nans<Op, T>::value) return x == x ? x : op_identity<Op, T>::value();
  else return x;
}

template <class Op> struct is_commutative_op : std::false_type {};
template <> struct is_commutative_op<plus_op> : std::true_type {};
template <> struct is_commutative_op<min_op> : std::true_type {};
template <> struct is_commutative_op<max_op> : std::true_type {};

// ---------------------------------------------------------------- what chains the tiles
// C: the type in which tile totals travel and a round's totals are added up; R: the running total over the
// rounds.  Both are the element type where the operator is exact and have more bits where sums of floats are
// rounded, so that the chain over thousands of tiles adds no error of its own: fp32 totals travel as doubles whose two
// lowest mantissa bits give way to the status (one 64-bit word); fp64 totals are summed in a pair of doubles from
// round to round (inside a round plain doubles do: their rounding is that of one round's sum, not of the total).
struct double_pair { double hi, lo; };
__device__ __forceinline__ double_pair add_to_pair(const double_pair& a, double b) {
  const double s = a.hi + b, bb = s - a.hi;
  double e = (a.hi - (s - bb)) + (b - bb);   // the rounding error of s (Knuth's two-sum)
  e += a.lo;
  double_pair r;
  r.hi = s + e;
  r.lo = e - (r.hi - s);
  if (!isfinite(r.hi) || (a.hi == 0.0 && b == 0.0)) { r.hi = s; r.lo = 0.0; }   // infinities stay, and so does the sign of zero
  return r;
}

template <class Chain> __device__ __forceinline__ typename Chain::C pipe_fold_round(const typename Chain::C (&v)[PIPE_SLOTS], int count);

template <class T, class Op> struct tile_chain {
  using C = T;
  using R = typename std::conditional<std::is_same<T, double>::value && std::is_same<Op, plus_op>::value, double_pair, T>::type;
  tile_state<T> ts;
  static size_t bytes(size_t tiles) { return tile_state<T>::bytes(tiles); }
  void bind(void* p, size_t tiles) { ts.bind(p, tiles); }
  __device__ static C identity() { return op_identity<Op, T>::value(); }
  __device__ static C lift(const T& x) { return x; }
  __device__ static T lower(const C& x) { return x; }
  __device__ static C join(const C& older, const C& newer) { return Op()(older, newer); }
  __device__ static R start(const C& x) { if constexpr (std::is_same<R, double_pair>::value) return R{x, 0.0}; else return x; }
  __device__ static R extend(const R& r, const C& x) { if constexpr (std::is_same<R, double_pair>::value) return add_to_pair(r, x); else return join(r, x); }
  __device__ static C value(const R& r) { if constexpr (std::is_same<R, double_pair>::value) return r.hi; else return r; }
  __device__ static C fold_round(const C (&v)[PIPE_SLOTS], int count) { return pipe_fold_round<tile_chain>(v, count); }
  __device__ void publish(size_t tile, unsigned status, const C& v) const { ts.publish(tile, status, v); }
  __device__ unsigned poll(size_t tile, C& v) const { return ts.poll(tile, v); }
  __device__ void publish_release(size_t tile, unsigned status, const C& v) const { ts.publish_release(tile, status, v); }
  __device__ unsigned poll_acquire(size_t tile, C& v) const { return ts.poll_acquire(tile, v); }
};
template <> struct tile_chain<float, plus_op> {
  using C = double;
  using R = double;
  unsigned long long* words;
  static size_t bytes(size_t tiles) { return align_up(tiles * 8, 256); }
  void bind(void* p, size_t) { words = static_cast<unsigned long long*>(p); }
  __device__ static C identity() { return -0.0; }
  __device__ static C lift(float x) { return (double)x; }
  __device__ static float lower(const C& x) { return (float)x; }
  __device__ static C join(const C& older, const C& newer) { return older + newer; }
  __device__ static R start(const C& x) { return x; }
  __device__ static R extend(const R& r, const C& x) { return r + x; }
  __device__ static C value(const R& r) { return r; }
  __device__ static C fold_round(const C (&v)[PIPE_SLOTS], int count) { return pipe_fold_round<tile_chain>(v, count); }
  __device__ void publish(size_t tile, unsigned status, const C& v) const {
    st_relaxed_u64(words + tile, ((unsigned long long)__double_as_longlong(v) & ~3ull) | status);
  }
  __device__ unsigned poll(size_t tile, C& v) const {
    const unsigned long long w = ld_relaxed_u64(words + tile);
    v = __longlong_as_double((long long)(w & ~3ull));
    return (unsigned)w & 3u;
  }
};

// ---------------------------------------------------------------- shared state of the pipeline
// P: what a warp's part of a tile is summarised to; C: what tiles are chained by.
template <class P, class C> struct pipe_state {
  unsigned long long full[PIPE_STAGES];      // the stage's tile has arrived
  unsigned long long empty[PIPE_STAGES];     // every compute warp is done with the stage
  unsigned long long summed[PIPE_STAGES];    // every compute warp has left its summary in part[]
  unsigned long long carried[PIPE_STAGES];   // carry[] holds what precedes the stage's tile
  C carry[PIPE_STAGES];
  P part[PIPE_STAGES][PIPE_WARPS];
  unsigned dead;                             // a wait of this CTA has run out
};

template <class S> __device__ __forceinline__ void pipe_init(S& st) {
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < PIPE_STAGES; ++s) {
      mbar_init(&st.full[s], 1);
      mbar_init(&st.empty[s], PIPE_WARPS);
      mbar_init(&st.summed[s], PIPE_WARPS);
      mbar_init(&st.carried[s], 1);
    }
    st.dead = 0;
    mbar_init_fence();
  }
  __syncthreads();
}

// Where a role is in its sequence of tiles: the tile, its ring stage and phase parity.
struct pipe_cursor {
  unsigned tile = blockIdx.x, stage = 0, parity = 0;
  __device__ __forceinline__ void next(unsigned steps = 1) {
    tile += steps * gridDim.x;
    stage += steps;
    if (stage >= PIPE_STAGES) { stage -= PIPE_STAGES; parity ^= 1; }
  }
};
template <class S> __device__ __forceinline__ bool pipe_dead(const S& st) { return __any_sync(FULL_MASK, *(const volatile unsigned*)&st.dead != 0); }

// One array's part of a tile, by the whole loader warp: returns the bytes that a bulk copy brings; what the
// last, partial tile has behind its last whole 16 bytes comes by ordinary loads, then `pad`.
template <class T, int ITEMS>
__device__ __forceinline__ unsigned pipe_tail_fill(T* dst, const T* src, size_t left, const T& pad) {
  if (left >= (size_t)ITEMS) return ITEMS * sizeof(T);
  constexpr unsigned VEC = 16 / sizeof(T);
  const unsigned bulk = (unsigned)(left * sizeof(T)) & ~15u, at = bulk / sizeof(T);
  if (lane_id() < VEC && at < ITEMS) dst[at + lane_id()] = at + lane_id() < left ? src[at + lane_id()] : pad;
  vec16 fill;
#pragma unroll
  for (unsigned k = 0; k < VEC; ++k) reinterpret_cast<T*>(&fill)[k] = pad;
  for (unsigned v = at / VEC + 1 + lane_id(); v < ITEMS / VEC; v += 32) reinterpret_cast<vec16*>(dst)[v] = fill;
  __syncwarp();
  return bulk;
}

// The same for a tile whose warps' parts lie 16 bytes apart in shared memory, so that a warp can compact its part in
// place at the distance from a 16-byte boundary that its output has: PIPE_WARPS parts of PART items, copied by one
// lane of the loader each.  bytes(left): what the copies of a tile with `left` items up to the input's end bring in all.
template <class T, int PART> struct pipe_parts {
  static constexpr unsigned STRIDE = PART * sizeof(T) + 16, BYTES = PIPE_WARPS * STRIDE;
  __device__ static unsigned part_bytes(size_t left, unsigned part) {
    const size_t first = (size_t)part * PART;
    if (left <= first) return 0;
    return left - first >= (size_t)PART ? PART * (unsigned)sizeof(T) : (unsigned)((left - first) * sizeof(T)) & ~15u;
  }
  __device__ static unsigned bytes(size_t left) {
    if (left >= (size_t)PART * PIPE_WARPS) return PART * PIPE_WARPS * (unsigned)sizeof(T);
    return (unsigned)(left * sizeof(T)) & ~15u;
  }
  // lane `part` of the loader, after the expect: its part's copy, and by ordinary loads what lies behind the last
  // whole 16 bytes of the input
  __device__ static void copy(unsigned char* stage, const T* tile, size_t left, unsigned part, unsigned long long* bar, unsigned long long policy) {
    const unsigned b = part_bytes(left, part);
    if (b) bulk_load(stage + part * STRIDE, tile + (size_t)part * PART, b, bar, policy);
  }
  __device__ static void ragged(unsigned char* stage, const T* tile, size_t left) {
    if (left >= (size_t)PART * PIPE_WARPS) return;
    const size_t i = (size_t)(((unsigned)(left * sizeof(T)) & ~15u) / sizeof(T)) + lane_id();
    if (lane_id() < 16 / (int)sizeof(T) && i < left) *reinterpret_cast<T*>(stage + (i / PART) * STRIDE + (i % PART) * sizeof(T)) = tile[i];
  }
  __device__ static T* part(unsigned char* stage, unsigned p) { return reinterpret_cast<T*>(stage + p * STRIDE); }
};

// The loader warp.  fill(stage, tile) brings the tile into the stage: the whole warp calls it, lane 0 arrives
// on st.full[stage] with the bytes it expects.
template <class S, class Fill>
__device__ __forceinline__ void pipe_loader(S& st, unsigned tiles, unsigned* err, Fill fill) {
  unsigned issued = 0;
  for (pipe_cursor cur; cur.tile < tiles; cur.next()) {
    pipe_wait(&st.empty[cur.stage], cur.parity ^ 1, &st.dead, err);
    if (pipe_dead(st)) break;
    __syncwarp();
    fill(cur.stage, cur.tile);
    ++issued;
  }
  // the CTA does not end before its bulk copies have landed
  for (unsigned i = issued > PIPE_STAGES ? issued - PIPE_STAGES : 0; i < issued; ++i)
    for (unsigned iter = 0; !mbar_try_wait(&st.full[i % PIPE_STAGES], (i / PIPE_STAGES) & 1) && iter < MBAR_SPIN_LIMIT; ++iter) {}
}

// Order between CTAs.  A descriptor is one word, stored and polled relaxed: its value is all that a CTA takes from another
// one.  Where the output goes over the input (ORDERED: the in-place partition) it must also order this CTA's stores behind
// the other CTAs' copies of what lay there: the publisher releases what its CTA has seen arrive, the folder acquires it.
//
// The publisher warp.  fold(part) turns the warps' summaries (lane w < PIPE_WARPS holds warp w's) into the tile's total, valid in lane 0.
template <bool ORDERED, class S, class Chain, class Fold>
__device__ __forceinline__ void pipe_publisher(S& st, const Chain& chain, unsigned tiles, unsigned* err, Fold fold) {
  for (pipe_cursor cur; cur.tile < tiles; cur.next()) {
    pipe_wait(&st.summed[cur.stage], cur.parity, &st.dead, err);
    if (pipe_dead(st)) return;
    const auto total = fold(st.part[cur.stage][lane_id() & (PIPE_WARPS - 1)]);
#ifdef TB200_TEST_HOOKS
    if (cur.tile == 0 && (reinterpret_cast<const ws_header*>(err)->flags & 1u)) continue;   // err points at the header's first word
#endif
    if (lane_id() == 0) {
      if constexpr (ORDERED) chain.publish_release(cur.tile, TILE_AGGREGATE, total); else chain.publish(cur.tile, TILE_AGGREGATE, total);
    }
  }
}

// The combination of the first `count` descriptors of a round, descriptor j * 32 + lane in v[j], for operators
// that commute: every lane folds its own, then a butterfly.  Result in every lane.
template <class Chain> __device__ __forceinline__ typename Chain::C pipe_fold_round(const typename Chain::C (&v)[PIPE_SLOTS], int count) {
  using C = typename Chain::C;
  C acc = Chain::identity();
#pragma unroll
  for (int j = 0; j < PIPE_SLOTS; ++j) if (j * 32 + lane_id() < count) acc = Chain::join(acc, v[j]);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) acc = Chain::join(acc, shfl_generic(acc, 0, 3, d));
  return acc;
}

// The folder warp.  last(total) is called by lane 0 of the last tile's CTA with everything up to the input's end.
template <bool ORDERED, class S, class Chain, class Last>
__device__ __forceinline__ void pipe_folder(S& st, const Chain& chain, unsigned tiles, const typename Chain::C& init, unsigned* err, Last last) {
  using C = typename Chain::C;
  const int lane = lane_id();
  auto poll = [&](size_t tile, C& value) { if constexpr (ORDERED) return chain.poll_acquire(tile, value); else return chain.poll(tile, value); };
  typename Chain::R running = Chain::start(init);   // everything before the current round
  for (pipe_cursor cur; cur.tile < tiles; cur.next()) {
    const unsigned base = cur.tile - blockIdx.x, round = tiles - base < gridDim.x ? tiles - base : gridDim.x;
    C v[PIPE_SLOTS];
    unsigned status[PIPE_SLOTS];
#pragma unroll
    for (int j = 0; j < PIPE_SLOTS; ++j) {
      status[j] = TILE_AGGREGATE; v[j] = Chain::identity();
      if (j * 32 + lane < round) status[j] = poll(base + j * 32 + lane, v[j]);
    }
    bool handed = false;
    for (unsigned iter = 0;; ++iter) {
      bool before_missing = false, missing = false;
#pragma unroll
      for (int j = 0; j < PIPE_SLOTS; ++j) {
        const bool m = status[j] == TILE_INVALID;
        missing |= m;
        before_missing |= m && j * 32 + lane <= blockIdx.x;
      }
      if (!handed && !__any_sync(FULL_MASK, before_missing)) {
        // the carry needs the CTAs before this one only (and this one's tile in its stage: what the stage held before is finished then)
        // That this CTA's own descriptor was there implies that its warps have summarised the tile, but by way of a relaxed word
        // in global memory.  Waiting for `summed` itself (it never has to) orders the warps' reads of each other's summaries,
        // and their stores over items that their neighbours looked at, behind the summaries.
        pipe_wait(&st.summed[cur.stage], cur.parity, &st.dead, err);
        __syncwarp();
        const C carry = Chain::value(Chain::extend(running, Chain::fold_round(v, (int)blockIdx.x)));
        if (lane == 0) { st.carry[cur.stage] = carry; mbar_arrive(&st.carried[cur.stage]); }
        handed = true;
      }
      if (!__any_sync(FULL_MASK, missing)) break;
      if (iter > SPIN_LIMIT && lane == 0) { *(volatile unsigned*)&st.dead = 1; record_error(err, ERR_LOOKBACK_TIMEOUT); }
      if (pipe_dead(st)) return;
      __nanosleep(PIPE_POLL_NS);
#pragma unroll
      for (int j = 0; j < PIPE_SLOTS; ++j) if (status[j] == TILE_INVALID) status[j] = poll(base + j * 32 + lane, v[j]);
    }
    running = Chain::extend(running, Chain::fold_round(v, PIPE_MAX_GRID));
    if (cur.tile == tiles - 1 && lane == 0) last(Chain::value(running));
  }
}

// A compute warp.  P summarise(stage, tile) for its part of a tile (valid in lane 0), later finish(stage, tile) once the
// stage's carry is known.  WRITES: finish also stores to the stage.
template <bool WRITES, class S, class Summarise, class Finish>
__device__ __forceinline__ void pipe_compute(S& st, unsigned tiles, unsigned* err, Summarise summarise, Finish finish) {
  const int lane = lane_id(), warp = (threadIdx.x >> 5) % PIPE_WARPS;
  pipe_cursor ahead, cur;
  ahead.next((threadIdx.x >> 5) / PIPE_WARPS);
  cur.next((threadIdx.x >> 5) / PIPE_WARPS);
  int open = 0;        // tiles summarised and not yet finished
  unsigned idle = 0;
  while (cur.tile < tiles) {
    // whichever can be done now: a tile that has arrived is summarised (the other CTAs wait for its total), else the
    // oldest one finished if its carry is known; a warp never sits on a ready carry because a load is late.
    if (ahead.tile < tiles && open <= PIPE_LOOKAHEAD && __all_sync(FULL_MASK, mbar_test(&st.full[ahead.stage], ahead.parity))) {
      __syncwarp();
      const auto part = summarise(ahead.stage, ahead.tile);
      if (lane == 0) { st.part[ahead.stage][warp] = part; mbar_arrive(&st.summed[ahead.stage]); }
      ahead.next(PIPE_GROUPS);
      ++open;
      idle = 0;
    } else if (open > 0 && __all_sync(FULL_MASK, mbar_test(&st.carried[cur.stage], cur.parity))) {
      __syncwarp();
      finish(cur.stage, cur.tile);
      if (WRITES) fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&st.empty[cur.stage]);
      cur.next(PIPE_GROUPS);
      --open;
      idle = 0;
    } else {
      if (++idle > SPIN_LIMIT && lane == 0) { *(volatile unsigned*)&st.dead = 1; record_error(err, ERR_LOOKBACK_TIMEOUT); }
      if (pipe_dead(st)) return;
      __nanosleep(20);
    }
  }
}

// A word per lane for each of a warp's open tiles, kept from a tile's summary to its end: tiles are finished in the order in which
// they were summarised, at most PIPE_LOOKAHEAD + 1 are open.
struct open_words {
  static_assert(PIPE_LOOKAHEAD == 1, "two tiles are open at most");
  unsigned even = 0, odd = 0, put_at = 0, taken = 0;
  __device__ __forceinline__ void put(unsigned w) { if (put_at & 1) odd = w; else even = w; ++put_at; }
  __device__ __forceinline__ unsigned take() { return taken++ & 1 ? odd : even; }
};

// Compacted output, by one warp: a run of items staged at the same distance from a 16-byte boundary as its
// place in the output leaves in 16-byte stores.  run_shift(dst): that distance in items.
template <class T> __device__ __forceinline__ unsigned run_shift(const T* dst) { return (unsigned)(reinterpret_cast<uintptr_t>(dst) & 15) / sizeof(T); }
// items [start, end) of `staged` to the same places of `base`, both 16-byte aligned; start <= 16 / sizeof(T)
template <class T> __device__ __forceinline__ void warp_store_run(T* base, const T* staged, unsigned start, unsigned end) {
  constexpr unsigned VEC = 16 / sizeof(T);
  const unsigned lane = lane_id();
  const unsigned piece0 = (start + VEC - 1) / VEC, piece1 = end / VEC;   // 16-byte pieces that belong to the run alone
  for (unsigned v = piece0 + lane; v < piece1; v += 32) store_stream16(base + v * VEC, reinterpret_cast<const vec16*>(staged)[v]);
  // the ragged ends: fewer than VEC items each
  if (lane < VEC) {
    if (lane >= start && lane < end && piece0 > 0) base[lane] = staged[lane];
  } else if (lane < 2 * VEC) {
    const unsigned i = piece1 * VEC + (lane - VEC);
    if (i < end && piece1 >= piece0) base[i] = staged[i];
  }
}

// Dynamic shared memory: PIPE_STAGES stages, 128-byte aligned by hand, then `extra` bytes.
constexpr size_t pipe_smem_bytes(size_t stage_bytes, size_t extra) { return PIPE_STAGES * stage_bytes + extra + 128; }
__device__ __forceinline__ unsigned char* pipe_align(unsigned char* raw) {
  return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 127) & ~(uintptr_t)127);
}

// CTAs of a pipeline kernel (0: the device cannot hold one).  `ready`: the caller's flags for this kernel, one per device.
template <class Kernel> size_t pipe_grid(Kernel kernel, size_t smem, size_t tiles, bool (&ready)[64]) {
  const device_info& di = current_device_info();
  int dev = 0;
  if (smem > (size_t)di.max_smem_optin || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!ready[dev]) {
    int per_sm = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, PIPE_BLOCK, smem) != cudaSuccess || per_sm < 1) { cudaGetLastError(); return 0; }
    ready[dev] = true;
  }
  size_t grid = (size_t)di.sm_count;
#ifdef TB200_TEST_HOOKS
  if (test_hook_flags() & 4u) grid = 2 * PIPE_MAX_GRID;
  else
#endif
  if (grid > (size_t)PIPE_MAX_GRID) grid = PIPE_MAX_GRID;
  return grid < tiles ? grid : tiles;
}

// Clears the header and the descriptors.
inline cudaError_t pipe_clear(void* ws, size_t bytes, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(ws, 0, bytes, stream);
#ifdef TB200_TEST_HOOKS
  if (e == cudaSuccess) e = cudaMemsetAsync(&static_cast<ws_header*>(ws)->flags, (int)(test_hook_flags() & 1u), 1, stream);
#endif
  return e;
}

template <class... Params, class... Args> cudaError_t pipe_launch(void (*kernel)(Params...), size_t grid, size_t smem, cudaStream_t stream, Args... args) {
  return cooperative_launch(kernel, grid, PIPE_BLOCK, smem, stream, args...);
}

}  // namespace tb200
