// Appends of the contraction and residual phases: a counter goes on past the
// capacity of its array (what does not fit is counted, not written), so it is
// as wide as the edges it may count, and a slot is tested in that width.  A
// 32-bit counter would come back into range, or below zero, after 2^31 edges.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define GB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define GB_HOST_DEVICE inline
#endif

namespace gb {

using append_count = unsigned long long;

// Slot of entry k of an append that got the counter value `first`, or -1 when
// it does not fit `cap` entries.
GB_HOST_DEVICE long long append_slot(append_count first, unsigned k, long long cap) {
  const append_count at = first + k;
  return at < (append_count)(cap > 0 ? cap : 0) ? (long long)at : -1;
}

}  // namespace gb
