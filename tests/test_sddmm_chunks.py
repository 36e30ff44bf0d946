"""CPU: the nonzeros that the SDDMM kernel's chunks load and store
(csrc/sddmm_chunks.h, the arithmetic that the kernel runs), compiled for the
host.  Every load lies in the CTA's own nonzeros, which are stored once each;
a CTA of empty rows, whose first nonzero may be the end of the arrays, touches
nothing."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rvvlasparse_b200", "csrc")
SHIM = r"""
#include "sddmm_chunks.h"
#include <cstdint>
// stored nonzeros in order; -1: a load out of range, -2: a nonzero out of order
extern "C" int64_t walk(int kb, int ke, int step) {
  using namespace rvvla;
  int64_t next = kb, chunks = 0;
  for (SddmmChunk ch = sddmm_first(kb, ke); ch.c0 < ke; ch.c0 += kSdChunk) {
    if (ch.c0 < 0 || ++chunks > 2 + ((int64_t)ke - kb) / kSdChunk) return -3;  // wrapped
    for (int k = 0; k < ch.end() + step; ++k) {
      const int64_t at = ch.load(k);
      if (at < kb || at >= ke) return -1;
      if (!ch.holds(k)) continue;
      if ((int64_t)ch.c0 + k != next++) return -2;
    }
  }
  return next;
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    d = tmp_path_factory.mktemp("sddmm")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "shim.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fwrapv", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", str(so)],
                   check=True)
    fn = C.CDLL(str(so)).walk
    fn.restype, fn.argtypes = C.c_int64, [C.c_int, C.c_int, C.c_int]
    return fn


@pytest.mark.parametrize("kb", [0, 1, 31, 32, 33, 100, 4095, 4096, 4097, 123456])
def test_loads_stay_in_the_rows_nonzeros(walk, kb):
    for n in [0, 1, 2, 31, 32, 33, 4095, 4096, 4097, 8192, 8193 + 31]:
        assert walk(kb, kb + n, 2048) == kb + n, n


@pytest.mark.parametrize("n", [1, 31, 32, 4095, 4096, 5000, 10 ** 7 + 3])
def test_largest_pattern(walk, n):
    """2^31 - 1 nonzeros: the step past the last chunk does not fit 32 bits."""
    end = 2 ** 31 - 1
    assert walk(end - n, end, 2048) == end
