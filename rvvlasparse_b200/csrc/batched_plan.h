// batched_plan.h — which warp of which CTA takes which slices of a batch's
// SELL matrices (batched.cu), host code without CUDA.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace rvvla {

struct SliceUnit {
  int32_t mat, slice;
  int64_t cost;  // columns, and a share for the slice itself
};

// Slices [first, end) of one matrix, by one warp.
struct alignas(16) BatchPart {
  int32_t mat, first, end, pad;
};

// Slices of one matrix by all 32 warps of a CTA: warp w takes
// [first[w], first[w + 1]).
constexpr int kSegWarps = 32;
struct BatchSeg {
  int32_t mat, first[kSegWarps + 1];
};

// The work of a batch, as parts or as segments.  Parts: warp w of CTA c takes
// parts[share[c * warps + w]] to parts[share[c * warps + w + 1] - 1].  Segments:
// CTA c takes segs[share[c]] to segs[share[c + 1] - 1].  busiest: the cost of
// the warp that has most to do.
struct SlicePlan {
  std::vector<BatchPart> parts;
  std::vector<BatchSeg> segs;
  std::vector<int32_t> share;
  int64_t busiest = 0;
};

// Cuts the slices of all SELL matrices, in order, into grid * pieces runs of
// equal cost and gives run r to CTA r mod grid, so that an SM's warps work on
// few matrices at a time: each(cta, u0, u1) for the units [u0, u1) of one matrix
// in a run.
template <class F>
void for_each_run(const std::vector<SliceUnit>& units, int grid, int pieces, F each) {
  int64_t total = 0, done = 0;
  for (const SliceUnit& u : units) total += u.cost;
  const int64_t runs = (int64_t)grid * pieces;
  size_t u0 = 0;
  for (int64_t r = 0; r < runs; ++r) {
    const double until = (double)total * (double)(r + 1) / (double)runs;
    size_t u1 = u0;
    while (u1 < units.size() && (r + 1 == runs || (double)done + 0.5 * (double)units[u1].cost < until))
      done += units[u1++].cost;
    while (u0 < u1) {
      size_t ue = u0;
      while (ue < u1 && units[ue].mat == units[u0].mat) ++ue;
      each((int)(r % grid), u0, ue);
      u0 = ue;
    }
  }
}

// Cuts the units [u0, u1) by cost into `warps` consecutive ranges, some of them
// empty where there are fewer units: each(w, a, b, cost of them).
template <class F>
void cut_by_cost(const std::vector<SliceUnit>& units, size_t u0, size_t u1, int warps, F each) {
  int64_t cost = 0, at = 0;
  for (size_t u = u0; u < u1; ++u) cost += units[u].cost;
  for (int w = 0; w < warps; ++w) {
    const size_t a = u0;
    const int64_t from = at;
    while (u0 < u1 && (w + 1 == warps || (double)at + 0.5 * (double)units[u0].cost < (double)cost * (w + 1) / warps))
      at += units[u0++].cost;
    each(w, a, u0, at - from);
  }
}

// Segments: each run's slices of a matrix are cut over the CTA's warps from
// warp 0 on.  Matrices of fewer slices than warps leave the other warps idle:
// of 20000 matrices of one slice, all 136 of a CTA are one warp's.
inline SlicePlan plan_segments(const std::vector<SliceUnit>& units, int grid, int pieces) {
  SlicePlan p;
  std::vector<std::vector<BatchSeg>> segs((size_t)grid);
  std::vector<int64_t> load((size_t)grid * kSegWarps, 0);
  for_each_run(units, grid, pieces, [&](int c, size_t u0, size_t u1) {
    BatchSeg sg = {};
    sg.mat = units[u0].mat;
    cut_by_cost(units, u0, u1, kSegWarps, [&](int w, size_t a, size_t b, int64_t cost) {
      sg.first[w] = a < u1 ? units[a].slice : units[u1 - 1].slice + 1;
      sg.first[w + 1] = b < u1 ? units[b].slice : units[u1 - 1].slice + 1;
      load[(size_t)c * kSegWarps + w] += cost;
    });
    segs[(size_t)c].push_back(sg);
  });
  p.share.assign(1, 0);
  for (const auto& list : segs) {
    p.segs.insert(p.segs.end(), list.begin(), list.end());
    p.share.push_back((int32_t)p.segs.size());
  }
  if (grid > 0) p.busiest = *std::max_element(load.begin(), load.end());
  return p;
}

// Parts: the ranges of a run's slices of a matrix (single slices, where there
// are fewer slices than warps) go to the warps that have least to do so far,
// the largest range first.
inline SlicePlan plan_parts(const std::vector<SliceUnit>& units, int grid, int pieces, int warps) {
  struct Range {
    size_t a, b;
    int64_t cost;
  };
  SlicePlan p;
  std::vector<std::vector<BatchPart>> parts((size_t)grid * warps);
  std::vector<int64_t> load((size_t)grid * warps, 0);
  std::vector<Range> ranges;
  std::vector<int> order((size_t)warps);
  for_each_run(units, grid, pieces, [&](int c, size_t u0, size_t u1) {
    int64_t* l = load.data() + (size_t)c * warps;
    auto give = [&](int w, size_t a, size_t b, int64_t cost) {
      const BatchPart q = {units[a].mat, units[a].slice, units[b - 1].slice + 1, 0};
      std::vector<BatchPart>& list = parts[(size_t)c * warps + w];
      if (!list.empty() && list.back().mat == q.mat && list.back().end == q.first) list.back().end = q.end;
      else list.push_back(q);
      l[w] += cost;
    };
    if (u1 - u0 < (size_t)warps) {
      for (size_t u = u0; u < u1; ++u) give((int)(std::min_element(l, l + warps) - l), u, u + 1, units[u].cost);
      return;
    }
    ranges.clear();
    cut_by_cost(units, u0, u1, warps, [&](int, size_t a, size_t b, int64_t cost) {
      if (a < b) ranges.push_back({a, b, cost});
    });
    std::stable_sort(ranges.begin(), ranges.end(), [](const Range& x, const Range& y) { return x.cost > y.cost; });
    for (int w = 0; w < warps; ++w) order[(size_t)w] = w;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return l[x] < l[y]; });
    for (size_t i = 0; i < ranges.size(); ++i) give(order[i], ranges[i].a, ranges[i].b, ranges[i].cost);
  });
  p.share.assign(1, 0);
  for (const auto& list : parts) {
    p.parts.insert(p.parts.end(), list.begin(), list.end());
    p.share.push_back((int32_t)p.parts.size());
  }
  if (!load.empty()) p.busiest = *std::max_element(load.begin(), load.end());
  return p;
}

}  // namespace rvvla
