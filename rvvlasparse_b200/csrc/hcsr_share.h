// hcsr_share.h — how many CTAs share a block row and which part of a window's
// COO stream each of them takes (hcsr_spmv.cu), in host and device code.
#pragma once

#include <algorithm>
#include <cstdint>

#include "host_device.h"

namespace rvvla {

// The nonzeros [lo, hi) of the stream, in rounds of `per` of them.
struct HcsrShare {
  int lo, hi;
  RVVLA_HD int rounds(int per) const { return (int)(((unsigned)(hi - lo) + (unsigned)per - 1u) / (unsigned)per); }
  // the first position of a warp's turn; unsigned, since the last round may
  // reach past 2^31 - 1
  RVVLA_HD unsigned first(int round, int per, int skip) const {
    return (unsigned)lo + (unsigned)round * (unsigned)per + (unsigned)skip;
  }
};

// Part `part` of `parts` of a stream of `total` nonzeros: multiples of 32, in
// order.  A stream holds every nonzero of up to 256 blocks when a block row is
// walked a second time, so the sums here need more than 32 bits.
RVVLA_HD inline HcsrShare hcsr_share(int total, int parts, int part) {
  const int64_t share = (((int64_t)total + parts - 1) / parts + 31) / 32 * 32;
  const int64_t lo = share * part < total ? share * part : total;
  const int64_t hi = lo + share < total ? lo + share : total;
  return {(int)lo, (int)hi};
}

constexpr int64_t kHSplitMax = 8;     // portable cluster size
constexpr int64_t kHSplitNz = 2048;   // nonzeros of a block row that a part keeps at least
constexpr int64_t kHSplitBlk = 96;    // nonzeros of a large block that a warp keeps at least

// Parts of a block row: as many as the free CTA slots give, fewer where a part
// would have too little of the block row, or its `warps` warps of the average
// block, if that has the `large` nonzeros with which blocks are cut by rows.
inline int hcsr_parts(int64_t b_m, int64_t b_n, int64_t nz, int64_t slots, int warps, int large) {
  int64_t s = std::min({slots / b_m, nz / (b_m * kHSplitNz), kHSplitMax});
  const int64_t block = nz / b_m / std::max<int64_t>(b_n, 1);
  if (block >= large) s = std::min(s, block / (warps * kHSplitBlk));
  return (int)std::max<int64_t>(1, s);
}

}  // namespace rvvla
