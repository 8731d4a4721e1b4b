// The rows of a unit that have pairs, as a warp of k_infect lists them
// (packed.cu).  A row's pairs have a word of their own: under the countdown rule
// rows of any length are listed, and a window may hold 2^30 contacts of one
// pair of nodes (repeated records are not merged in unsorted windows).
// Header-only so that a host-side test can compile it without the CUDA runtime.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define RP_HD __host__ __device__ __forceinline__
#else
#define RP_HD inline
#endif

namespace rp {

constexpr int kUnitRows = 128;  // most rows of a unit

struct UnitRows {
  int32_t beg[kUnitRows];  // their first pairs
  int32_t len[kUnitRows];  // their pairs
  uint8_t row[kUnitRows];  // row (or list entry) in the unit
  static_assert(kUnitRows <= 256, "a row of the unit in a byte");

  RP_HD void put(int pos, int r, int32_t first, int32_t pairs) {
    beg[pos] = first;
    len[pos] = pairs;
    row[pos] = (uint8_t)r;
  }
};

}  // namespace rp
