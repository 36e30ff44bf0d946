"""CPU: the shares of a batch's SELL slices (csrc/batched_plan.h, compiled for
the host): every slice goes to one warp, and in parts no warp has more than twice
the mean and a slice to do, whatever the matrices' sizes."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rvvlasparse_b200", "csrc")
SHIM = r"""
#include "batched_plan.h"
using namespace rvvla;
// (warp, matrix, first, end) in the order of a warp's work
static int64_t k, cap_;
static int32_t* out_;
static void put(int w, int m, int a, int b) {
  if (a < b && k < cap_) out_[4 * k] = w, out_[4 * k + 1] = m, out_[4 * k + 2] = a, out_[4 * k + 3] = b;
  k += a < b;
}
extern "C" int64_t plan(int64_t n, const int32_t* mat, const int32_t* slice, const int64_t* cost, int grid, int pieces,
                        int warps, int64_t cap, int32_t* out, int64_t* busiest) {
  std::vector<SliceUnit> u;
  for (int64_t i = 0; i < n; ++i) u.push_back({mat[i], slice[i], cost[i]});
  k = 0, cap_ = cap, out_ = out;
  const SlicePlan p = warps ? plan_parts(u, grid, pieces, warps) : plan_segments(u, grid, pieces);
  *busiest = p.busiest;
  if (p.share.size() != (size_t)grid * (warps ? warps : 1) + 1 || p.share[0] != 0) return -1;
  if (p.share.back() != (int64_t)(warps ? p.parts.size() : p.segs.size())) return -2;
  for (int c = 0; !warps && c < grid; ++c)
    for (int i = p.share[c]; i < p.share[c + 1]; ++i)
      for (int w = 0; w < kSegWarps; ++w) put(c * kSegWarps + w, p.segs[i].mat, p.segs[i].first[w], p.segs[i].first[w + 1]);
  for (int w = 0; w < grid * warps; ++w)
    for (int i = p.share[w]; i < p.share[w + 1]; ++i) put(w, p.parts[i].mat, p.parts[i].first, p.parts[i].end);
  return k;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("batched")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "shim.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).plan
    fn.restype = C.c_int64
    fn.argtypes = [C.c_int64] + [C.c_void_p] * 3 + [C.c_int] * 3 + [C.c_int64, C.c_void_p, C.c_void_p]

    def call(mat, sl, cost, grid, pieces, warps):
        out, busiest = np.zeros((len(mat) + grid * 32, 4), np.int32), C.c_int64(-1)
        k = fn(len(mat), mat.ctypes.data, sl.ctypes.data, cost.ctypes.data, grid, pieces, warps, len(out), out.ctypes.data,
               C.byref(busiest))
        assert 0 <= k <= len(out)
        return out[:k], busiest.value

    return call


def _load(plan, counts, cost, grid, pieces, warps):
    """Each warp's cost (warps 0: the segments'), every slice found once."""
    mat = np.repeat(np.arange(len(counts)), counts).astype(np.int32)
    sl = np.concatenate([np.arange(k) for k in counts] + [np.zeros(0)]).astype(np.int32)
    cost = np.ascontiguousarray(cost, np.int64)
    start = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    seen, load = np.zeros(len(mat), int), np.zeros(grid * (warps or 32), np.int64)
    work, busiest = plan(mat, sl, cost, grid, pieces, warps)
    for w, m, a, b in work:
        assert 0 <= a < b <= counts[m]
        seen[start[m] + a:start[m] + b] += 1
        load[w] += cost[start[m] + a:start[m] + b].sum()
    assert (seen == 1).all() and busiest == load.max()
    return load


def _check(plan, counts, cost, grid=148, pieces=1, warps=32):
    load = _load(plan, counts, cost, grid, pieces, warps)
    most = np.max(cost, initial=0)
    assert load.max() <= 2 * load.mean() + most, (load.max(), load.mean(), most)


@pytest.mark.parametrize("warps,pieces", [(32, 1), (16, 1), (16, 4)])
@pytest.mark.parametrize("slices,count", [(1, 20000), (2, 10000), (4, 8000), (8, 4000), (31, 1000), (33, 1000), (63, 1000), (64, 1000),
                                          (127, 500), (128, 500), (140, 500), (2048, 20)])
def test_equal_matrices(plan, slices, count, warps, pieces):
    _check(plan, [slices] * count, np.full(slices * count, 20), pieces=pieces, warps=warps)


@pytest.mark.parametrize("warps,pieces", [(32, 1), (16, 4)])
def test_uneven_matrices(plan, warps, pieces):
    rng = np.random.default_rng(3)
    counts = np.exp(rng.uniform(0, np.log(200), 3000)).astype(int)
    _check(plan, counts, rng.integers(2, 100, counts.sum()), pieces=pieces, warps=warps)
    # wide slices first in every matrix (sorted rows), and one wide kind in eight
    cost = np.concatenate([np.sort(rng.integers(2, 200, k))[::-1] for k in counts])
    _check(plan, counts, cost, pieces=pieces, warps=warps)
    _check(plan, [1] * 16000, np.where(np.arange(16000) % 8 == 0, 200, 3), pieces=pieces, warps=warps)


@pytest.mark.parametrize("counts", [[], [0, 0], [1], [0, 1, 0], [3, 0, 5], [1] * 147, [1] * 149, [5000]])
def test_few_slices(plan, counts):
    _check(plan, counts, np.full(sum(counts), 9))


def test_segments(plan):
    """The other form: complete too, level for large matrices, one warp's work
    for matrices of one slice."""
    rng = np.random.default_rng(5)
    counts = rng.integers(400, 2000, 200)
    load = _load(plan, counts, rng.integers(2, 60, counts.sum()), 148, 1, 0)
    assert load.max() <= 1.2 * load.mean()
    load = _load(plan, [1] * 20000, np.full(20000, 20), 148, 1, 0)
    assert load.max() > 30 * load.mean()
    for counts in ([], [1], [0, 3, 0], [31, 32, 33]):
        _load(plan, counts, np.full(sum(counts), 9), 148, 1, 0)
