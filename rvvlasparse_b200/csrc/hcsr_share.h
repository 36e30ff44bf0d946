// hcsr_share.h — the part of a window's COO stream that one CTA of a block row
// takes (hcsr_spmv.cu), in host and device code.
#pragma once

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

}  // namespace rvvla
