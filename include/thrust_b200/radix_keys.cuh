// Keys as the radix sorts see them and the ranking of their digits, shared by the general sort (radix_sort.cuh) and the small
// one (cluster_sort.cuh).
//
// Key order is defined on an unsigned code of the key: unsigned keys unchanged, signed keys
// with the sign bit flipped, IEEE floats with all bits flipped when negative and the sign bit
// flipped otherwise (the encoders of thrust/system/detail/sequential/stable_radix_sort.inl:54-138);
// descending order complements the code.
#pragma once
#include "common.cuh"

namespace tb200 {

constexpr int RADIX_BITS = 8;
constexpr int RADIX_BINS = 256;

enum key_kind : int { KEY_UNSIGNED = 0, KEY_SIGNED = 1, KEY_FLOAT = 2 };

struct key_coding {
  int kind; int descending;
};

// Digit `shift / 8` of the key's order-preserving unsigned code.  For integer keys the code
// differs from the raw bits by a constant, so the digit is the raw byte XOR `dmask` (the matching
// byte of that constant); float keys first flip all bits of negative values.
template <class UK> __host__ __device__ __forceinline__ unsigned digit_mask(key_coding c, int shift) {
  constexpr int B = 8 * sizeof(UK);
  UK m = c.descending ? (UK)~(UK)0 : (UK)0;
  if (c.kind != KEY_UNSIGNED) m ^= (UK)1 << (B - 1);
  return (unsigned)(m >> shift) & 0xffu;
}
template <class UK> __device__ __forceinline__ UK float_digits(UK k) {   // negative: flip the non-sign bits too
  constexpr int B = 8 * sizeof(UK);
  using SK = typename std::make_signed<UK>::type;
  return k ^ ((UK)((SK)k >> (B - 1)) & (UK)~((UK)1 << (B - 1)));
}
template <bool IS_FLOAT, class UK> __device__ __forceinline__ unsigned key_digit(UK k, int shift, unsigned dmask) {
  if (IS_FLOAT) k = float_digits(k);
  return ((unsigned)(k >> shift) & 0xffu) ^ dmask;
}

#ifndef TB200_SWEEP_LOOP_MAX
#define TB200_SWEEP_LOOP_MAX 6      // rows with more colliding lanes than this are ranked with ballots
#endif

// Ranks one row of 32 items, one per lane, on the warp's private counters in shared memory: adds 1 to the counter of this
// lane's digit and returns the item's place behind what the counter held before the row, in lane order.  Every lane adds 1
// and then reads the counter back: `old` is some slot of the digit's group in this row, `now - old > 1` tells all members
// of a group of two or more lanes, except the one that drew the last slot, that they collided.  Lanes that did not collide
// are done (rank = old).  Groups are then put in lane order one at a time: the highest colliding lane announces
// its digit, one ballot finds its group, each member takes base + (members in lower lanes).  With 256 bins and 32 lanes
// a row has about two groups, which costs half the instructions of finding every lane's peers with one ballot per digit
// bit; rows with more than TB200_SWEEP_LOOP_MAX colliding lanes (skewed digits, a padded tile), and all rows of digits of up to
// four bits, take the ballots.  The result does not depend on the order in which the hardware serves the atomics.
template <int BITS> __device__ __forceinline__ unsigned warp_rank(unsigned* counters, unsigned d, unsigned lanemask_ge) {
  const unsigned old = atomicAdd(&counters[d], 1u);
  __syncwarp();   // every lane's increment precedes every lane's read
  const unsigned now = *reinterpret_cast<volatile unsigned*>(&counters[d]);
  unsigned pending = __ballot_sync(FULL_MASK, now - old > 1u);
  unsigned rank = old;
  if (BITS > 4 ? __popc(pending) <= TB200_SWEEP_LOOP_MAX : pending == 0) {
    while (pending) {
      const unsigned dsrc = __shfl_sync(FULL_MASK, d, 31 - __clz(pending));
      const unsigned peers = __ballot_sync(FULL_MASK, d == dsrc);
      if (d == dsrc) rank = now - __popc(peers & lanemask_ge);   // base + members in lower lanes
      pending &= ~peers;
    }
  } else {
    unsigned peers = FULL_MASK;
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
      const bool bit = (d >> b) & 1;
      const unsigned vote = __ballot_sync(FULL_MASK, bit);
      peers &= bit ? vote : ~vote;
    }
    rank = now - __popc(peers & lanemask_ge);
  }
  return rank;
}

// Turns per-warp digit counts into places, by the first 256 threads of a CTA (thread t: digit t); two barriers of the CTA lie inside, so
// every thread calls it.  hist: [WARPS][256], on return each warp's first place of each digit inside the CTA.  publish(count) is called
// with the CTA's count of the digit as soon as that is known; returns the digit's first place.  All loads of a step are
// issued before the first result is used: one after the other they are much of a small sort's digit place.
template <int WARPS, class Publish>
__device__ __forceinline__ unsigned stack_digits(unsigned* hist, unsigned (&s_scan)[RADIX_BINS / 32], Publish publish) {
  const int t = threadIdx.x, warp = t >> 5;
  unsigned first[WARPS], run = 0, place = 0;
  if (t < RADIX_BINS) {
#pragma unroll
    for (int w = 0; w < WARPS; ++w) first[w] = hist[w * RADIX_BINS + t];
#pragma unroll
    for (int w = 0; w < WARPS; ++w) { const unsigned c = first[w]; first[w] = run; run += c; }
    publish(run);
    place = warp_inclusive_scan(run, plus_op());
    if (lane_id() == 31) s_scan[warp] = place;
    place -= run;
  }
  __syncthreads();
  if (t < RADIX_BINS) {
#pragma unroll
    for (int w = 0; w < RADIX_BINS / 32; ++w) { const unsigned c = s_scan[w]; place += w < warp ? c : 0u; }
#pragma unroll
    for (int w = 0; w < WARPS; ++w) hist[w * RADIX_BINS + t] = first[w] + place;
  }
  __syncthreads();
  return place;
}

}  // namespace tb200
