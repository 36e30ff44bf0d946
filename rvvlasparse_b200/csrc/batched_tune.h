// batched_tune.h — how the batched autotuner (batched.cu) chooses each matrix's
// layout from measured times, host code without CUDA.
#pragma once

#include <cstddef>
#include <cstdint>
#include <numeric>
#include <vector>

namespace rvvla {

struct TuneCand {
  int32_t mode, param;  // mode: 0 CSR, 1 SELL
};

// Batches of up to this time in all are compared whole (a second launch, 4 to 8
// us, counts for little in longer ones).
constexpr double kTuneWholeMs = 0.1;

// Times every candidate on each group of matrices and gives the group its
// fastest.  time(ids, cands, &ms) times the matrices `ids` with a candidate each
// and returns 0, or a status that ends the search.  Picks of both layouts make
// two launches, which groups timed by themselves do not show (16 matrices of 1K to
// 4K rows, fp64, k = 1: 22 us with 7 of them in SELL, 14 with all in CSR): a
// short batch is then timed whole, so and with each group's fastest CSR and
// fastest SELL candidate.  For longer ones that would only lengthen the tuning (256
// matrices of 1K to 64K rows, k = 1, of 258 us: 0.4 s for the three plans).  The cands hold both layouts.
template <class Time>
int tune_layouts(const std::vector<std::vector<int64_t>>& groups, int64_t count, const std::vector<TuneCand>& cands,
                 Time time, std::vector<TuneCand>& out, double* total) {
  std::vector<TuneCand> choice[3];  // per matrix: the fastest, the fastest CSR, the fastest SELL candidate
  for (auto& c : choice) c.resize((size_t)count);
  bool used[2] = {false, false};
  double sum = 0.0;
  for (const auto& grp : groups) {
    if (grp.empty()) continue;
    double best[2] = {1e30, 1e30};
    TuneCand pick[2] = {cands.front(), cands.back()};
    for (const TuneCand& c : cands) {
      double ms = 0.0;
      if (const int rc = time(grp, std::vector<TuneCand>(grp.size(), c), &ms)) return rc;
      if (ms < best[c.mode]) {
        best[c.mode] = ms;
        pick[c.mode] = c;
      }
    }
    const int w = best[1] < best[0] ? 1 : 0;
    for (int64_t i : grp) {
      choice[0][(size_t)i] = pick[w];
      choice[1][(size_t)i] = pick[0];
      choice[2][(size_t)i] = pick[1];
    }
    used[w] = true;
    sum += best[w];
  }
  int w = 0;
  if (used[0] && used[1] && sum <= kTuneWholeMs) {
    std::vector<int64_t> all((size_t)count);
    std::iota(all.begin(), all.end(), (int64_t)0);
    sum = 1e30;
    for (int c = 0; c < 3; ++c) {
      double ms = 0.0;
      if (const int rc = time(all, choice[c], &ms)) return rc;
      if (ms < sum) {
        sum = ms;
        w = c;
      }
    }
  }
  out = choice[w];
  *total = sum;
  return 0;
}

}  // namespace rvvla
