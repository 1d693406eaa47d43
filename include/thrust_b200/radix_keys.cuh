// Keys as the radix sorts see them, shared by the general sort (radix_sort.cuh) and the small one (cluster_sort.cuh).
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

}  // namespace tb200
