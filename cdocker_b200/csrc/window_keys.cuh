// window_keys.cuh -- keys of the window minimum: (energy, linear index) as one 64-bit value whose
// order is the energy's, then the index's (x-major first), and the smallest or two smallest of them.
#pragma once
#include <cuda_runtime.h>

namespace cdk {

__device__ __forceinline__ unsigned int order_key(float f) {
  unsigned int u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(unsigned int k) {
  unsigned int u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

// keep the two smallest keys (b1 < b2) of a stream of distinct keys
__device__ __forceinline__ void top2_insert(unsigned long long k, unsigned long long& b1, unsigned long long& b2) {
  // most candidates lose to the current second-smallest on the energy bits alone (one 32-bit
  // compare); the 64-bit order decides the rest
  if ((unsigned int)(k >> 32) > (unsigned int)(b2 >> 32)) return;
  if (k < b1) {
    b2 = b1;
    b1 = k;
  } else if (k < b2) {
    b2 = k;
  }
}
// merge another pair of two smallest into (b1, b2)
__device__ __forceinline__ void top2_merge(unsigned long long o1, unsigned long long o2, unsigned long long& b1,
                                           unsigned long long& b2) {
  const unsigned long long n1 = o1 < b1 ? o1 : b1;
  const unsigned long long hi = o1 < b1 ? b1 : o1;
  const unsigned long long lo2 = o2 < b2 ? o2 : b2;
  b2 = hi < lo2 ? hi : lo2;
  b1 = n1;
}

// Candidate energies e at linear index lin, into a thread's smallest key (b1) or two smallest
// keys (b1, b2). thr is the float of the largest key kept (+inf while a slot is empty): a value
// strictly above it (as floats, the same order as the keys) cannot enter and is rejected before
// its key is built; equal values, NaN and signed zeros take the exact 64-bit key path.
template <bool TOP2>
__device__ __forceinline__ void keep_min(float e, unsigned int lin, unsigned long long& b1, unsigned long long& b2,
                                         float& thr) {
  if (e > thr) return;
  const unsigned long long k = ((unsigned long long)order_key(e) << 32) | lin;
  if constexpr (TOP2) {
    top2_insert(k, b1, b2);
    thr = b2 == ~0ull ? INFINITY : key_to_float((unsigned int)(b2 >> 32));
  } else {
    if (k < b1) {
      b1 = k;
      thr = key_to_float((unsigned int)(k >> 32));
    }
  }
}

// smallest 64-bit key of the warp: redux on the high words, then on the low words of the lanes
// holding the smallest high word
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
  const unsigned int hi = __reduce_min_sync(0xffffffffu, (unsigned int)(k >> 32));
  const unsigned int lo = __reduce_min_sync(0xffffffffu, (unsigned int)(k >> 32) == hi ? (unsigned int)k : 0xffffffffu);
  return ((unsigned long long)hi << 32) | lo;
}
// the warp's two smallest keys from every lane's (b1 < b2) of distinct keys: the smallest b1,
// then the smallest of (b2 on the lane holding it, b1 elsewhere)
template <bool TOP2>
__device__ __forceinline__ void warp_keep_min(unsigned long long& b1, unsigned long long& b2) {
  const unsigned long long k1 = warp_min_key(b1);
  if constexpr (TOP2) b2 = warp_min_key(b1 == k1 ? b2 : b1);
  b1 = k1;
}

}  // namespace cdk
