"""CPU: the batched autotuner's choice of layouts (csrc/batched_tune.h, compiled
for the host) under a timer that knows what each matrix costs in each layout and
what a launch costs: never slower than all matrices in one layout where the batch
is short, each group's fastest where it is long."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rvvlasparse_b200", "csrc")
SHIM = r"""
#include "batched_tune.h"
using namespace rvvla;
// cost[i][c]: matrix i with candidate c (CSR 1, 8; SELL 32, 256); a launch per layout present
extern "C" int tune(int count, const int32_t* group, const double* cost, double launch, int fail_at, int32_t* mode,
                    double* total, int* plans) {
  const std::vector<TuneCand> cands = {{0, 1}, {0, 8}, {1, 32}, {1, 256}};
  std::vector<std::vector<int64_t>> groups(8);
  for (int i = 0; i < count; ++i) groups[group[i]].push_back(i);
  std::vector<TuneCand> out;
  int n = 0;
  const int rc = tune_layouts(groups, count, cands, [&](const std::vector<int64_t>& ids, const std::vector<TuneCand>& of, double* ms) {
    bool used[2] = {false, false};
    *ms = 0.0;
    for (size_t i = 0; i < ids.size(); ++i) {
      used[of[i].mode] = true;
      const int c = of[i].param == 1 ? 0 : of[i].param == 8 ? 1 : of[i].param == 32 ? 2 : 3;
      *ms += cost[4 * ids[i] + c];
    }
    *ms += launch * (used[0] + used[1]);
    return ++n == fail_at ? 7 : 0;
  }, out, total);
  for (size_t i = 0; i < out.size(); ++i) mode[i] = out[i].mode;
  *plans = n;
  return rc;
}
"""


@pytest.fixture(scope="module")
def tune(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "shim.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).tune

    def call(group, cost, launch, fail_at=0):
        group, cost = np.ascontiguousarray(group, np.int32), np.ascontiguousarray(cost, np.float64)
        mode, total, plans = np.full(len(group), -1, np.int32), C.c_double(-1), C.c_int(0)
        rc = fn(len(group), group.ctypes.data_as(C.c_void_p), cost.ctypes.data_as(C.c_void_p), C.c_double(launch), fail_at,
                mode.ctypes.data_as(C.c_void_p), C.byref(total), C.byref(plans))
        return rc, mode, total.value, plans.value

    return call


@pytest.mark.parametrize("seed", range(8))
@pytest.mark.parametrize("scale", [0.001, 0.1])  # ms per matrix: batches well below and above a tenth of a millisecond
def test_layouts(tune, seed, scale):
    rng = np.random.default_rng(seed)
    count, launch = 24, 0.006
    group = rng.integers(0, 3, count)
    group[:3] = [0, 1, 2]
    cost = rng.uniform(0.9, 1.1, (count, 4)) * scale
    rc, mode, total, plans = tune(group, cost, launch)
    per = [[cost[group == g, c].sum() for c in range(4)] for g in range(3)]
    csr, sell = (sum(min(p[2 * i:2 * i + 2]) for p in per) for i in (0, 1))
    best = [min(range(4), key=lambda c: p[c]) >= 2 for p in per]
    assert rc == 0
    if scale == 0.1:  # long: the groups' own picks
        assert (mode == np.array(best)[group]).all() and plans == 12
    elif len(set(best)) == 1:
        assert plans == 12
    else:
        mixed = sum(min(p) for p in per) + 2 * launch
        assert plans == 15 and total == pytest.approx(min(mixed, csr + launch, sell + launch))
        used = set(mode.tolist())
        assert (len(used) == 2) == (mixed < min(csr, sell) + launch)


def test_second_launch_counts(tune):
    """One group a little faster in SELL: all CSR, for the launch that saves."""
    cost = np.array([[2.0, 2, 3, 3]] * 8 + [[2.0, 2, 1.9, 1.9]] * 8) * 1e-3
    rc, mode, _, _ = tune([0] * 8 + [1] * 8, cost, 0.006)
    assert rc == 0 and (mode == 0).all()


def test_errors_end_the_search(tune):
    for at in (1, 6, 9):
        rc, _, _, plans = tune([0, 1], np.array([[1.0, 2, 3, 4], [4, 3, 2, 1]]) * 1e-3, 0.006, at)
        assert rc == 7 and plans == at
