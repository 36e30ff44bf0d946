// sddmm_chunks.h — the index arithmetic of sddmm_kernel (adjoint.cu), in host
// and device code: which nonzeros a CTA's chunks read and write.
#pragma once

#include <cstdint>

#include "host_device.h"

namespace rvvla {

constexpr int kSdChunk = 4096;  // nonzeros per pass over the row-start bitmap

// One chunk of a CTA's nonzeros [kb, ke): its slots k = 0 .. end() - 1 stand
// for the nonzeros c0 + k.  Chunks start at multiples of 32, so the first one
// may have slots before kb.
// c0 has 64 bits: the step past the last chunk of 2^31 - 1 nonzeros leaves 32.
struct SddmmChunk {
  int64_t c0;
  int kb, ke;
  RVVLA_HD int end() const { return ke - c0 < kSdChunk ? (int)(ke - c0) : kSdChunk; }
  // the nonzero that slot k loads: slots outside [kb, ke) repeat its first or last
  RVVLA_HD int64_t load(int k) const {
    const int64_t j = c0 + (k < end() - 1 ? k : end() - 1);
    return j > kb ? j : kb;
  }
  RVVLA_HD bool holds(int k) const { return k < end() && c0 + k >= kb; }
};

// The first chunk.  A CTA whose rows are all empty has none: its kb may be the
// end of the arrays, and a chunk aligned below kb would load from there.
RVVLA_HD inline SddmmChunk sddmm_first(int kb, int ke) { return {kb < ke ? kb / 32 * 32 : ke, kb, ke}; }

}  // namespace rvvla
