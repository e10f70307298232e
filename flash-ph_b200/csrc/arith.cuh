// Integer arithmetic at the edge of its range, apart from the kernels so that
// the host can run it too.
#pragma once
#include "common.cuh"

namespace ph {

// The middle of two positions lo <= hi. An adjacency has up to 2^31 - 2
// entries, so the sum of two of its positions does not fit 32 bits.
__host__ __device__ __forceinline__ int midpoint(int lo, int hi) { return lo + ((hi - lo) >> 1); }

// First position in [lo, hi) whose entry is not below x (hi where all are); a
// is anything that is indexed as an array.
template <typename Array>
__host__ __device__ __forceinline__ int lower_bound_i32(const Array& a, int lo, int hi, i32 x) {
  while (lo < hi) {
    const int mid = midpoint(lo, hi);
    if (a[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

}  // namespace ph
