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
template <bool IS_FLOAT, class UK> __device__ __forceinline__ unsigned key_digit(UK k, int shift, unsigned dmask) {
  constexpr int B = 8 * sizeof(UK);
  if (IS_FLOAT) {
    using SK = typename std::make_signed<UK>::type;
    k ^= (UK)((SK)k >> (B - 1)) & (UK)~((UK)1 << (B - 1));   // negative: flip the non-sign bits too
  }
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

}  // namespace tb200
