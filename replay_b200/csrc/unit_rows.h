// The rows of a unit that have pairs, as a warp of k_infect lists them
// (packed.cu).  kAnyLength: under the countdown rule rows of any length are
// listed, and a window may hold 2^30 contacts of one pair of nodes, so that a
// row's number of pairs has a word of its own.  Geometric rows listed here have
// at most 48 pairs, which share a word with the row (the separate arrays cost
// N = 1,000 with 1,000 replicas 2%; the countdown rule gained 5% from them).
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

template <bool kAnyLength>
struct UnitRows {
  int32_t word[kUnitRows];  // row (or list entry) in the unit | pairs << 7
  int32_t beg[kUnitRows];   // first pairs
  static_assert(kUnitRows <= 128, "a row of the unit in 7 bits");

  RP_HD void put(int pos, int r, int32_t first, int32_t pairs) {
    word[pos] = r | pairs << 7;
    beg[pos] = first;
  }
  RP_HD void get(int pos, int &r, int32_t &first, int32_t &pairs) const {
    r = word[pos] & 127;
    pairs = word[pos] >> 7;
    first = beg[pos];
  }
};

template <>
struct UnitRows<true> {
  int32_t len[kUnitRows];  // numbers of pairs
  int32_t beg[kUnitRows];
  uint8_t row[kUnitRows];

  RP_HD void put(int pos, int r, int32_t first, int32_t pairs) {
    len[pos] = pairs;
    beg[pos] = first;
    row[pos] = (uint8_t)r;
  }
  RP_HD void get(int pos, int &r, int32_t &first, int32_t &pairs) const {
    r = row[pos];
    pairs = len[pos];
    first = beg[pos];
  }
};

}  // namespace rp
