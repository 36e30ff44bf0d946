"""CPU: the shares of a COO stream and the positions of their rounds
(csrc/hcsr_share.h, the arithmetic that the HCSR kernel runs), compiled for
the host: the parts follow each other and cover the stream, up to 2^31 - 1
nonzeros."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rvvlasparse_b200", "csrc")
SHIM = r"""
#include "hcsr_share.h"
extern "C" void share(int total, int parts, int part, int per, int64_t* out) {
  const rvvla::HcsrShare s = rvvla::hcsr_share(total, parts, part);
  const int r = s.rounds(per);
  out[0] = s.lo, out[1] = s.hi, out[2] = r, out[3] = s.first(r > 0 ? r - 1 : 0, per, 0), out[4] = s.first(r, per, -1);
}
extern "C" int parts(int64_t b_m, int64_t b_n, int64_t nz, int64_t slots) {
  return rvvla::hcsr_parts(b_m, b_n, nz, slots, 8, 1024);
}
"""


@pytest.fixture(scope="module")
def share(tmp_path_factory):
    d = tmp_path_factory.mktemp("hcsr")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "shim.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fwrapv", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))

    def call(total, parts, part, per=512):
        out = (C.c_int64 * 5)()
        lib.share(total, parts, part, per, out)
        return list(out)

    call.parts = lambda *a: lib.parts(*(C.c_int64(v) for v in a))
    return call


@pytest.mark.parametrize("parts", range(1, 9))
@pytest.mark.parametrize("total", [0, 1, 31, 32, 33, 511, 512, 513, 262143, 2 ** 31 - 513, 2 ** 31 - 32, 2 ** 31 - 7, 2 ** 31 - 1])
def test_parts_cover_the_stream(share, total, parts):
    at = 0
    for p in range(parts):
        lo, hi, rounds, first, last = share(total, parts, p)
        assert lo == at and lo <= hi <= total
        assert lo == hi or lo % 32 == 0
        assert rounds == -(-(hi - lo) // 512)
        if hi > lo:  # the last round begins before the end and reaches it
            assert lo <= first < hi <= last + 1 < hi + 512
        at = hi
    assert at == total


SLOTS = 592 * 7 // 8


@pytest.mark.parametrize("b_m,b_n,nz,want", [
    (50, 50, 1_600_000, 8),  # power law: small blocks, as many as the cluster takes
    (90, 90, 13_940_000, 2),  # random rows: the average block is large
    (125, 125, 20_000_000, 1),
    (50, 50, 4_000_000, 2),
    (4, 1, 8_000_000, 8),  # few, very large blocks
    (501, 501, 19_600_000, 1),  # no free slots
    (30, 30, 2048 * 30 - 1, 1),  # too little for a second part
    (1, 0, 0, 1), (1, 1, 0, 1), (1, 1, 2 ** 31 - 1, 8)])
def test_parts_of_a_block_row(share, b_m, b_n, nz, want):
    assert share.parts(b_m, b_n, nz, SLOTS) == want
