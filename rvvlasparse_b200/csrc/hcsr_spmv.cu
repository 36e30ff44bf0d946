// hcsr_spmv.cu — y = alpha*A*x + beta*y for spMtxHCSR on sm_100a.
//
// Reference: src/scalar/spmv_mtx_hcsr.cpp:22-134.  The reference walks a
// block row's blocks in block-column order and adds every block's
// contribution into y[block row]: a CSR block (kind 1) adds one row sum per
// row, a COO block (any other kind) adds one product per nonzero.  Any R and
// C are accepted (the only limits are the format's: uint16 local columns,
// 30-bit row_ptr offsets).
//
// GPU mapping.  A block row belongs to one CTA of 8 warps, or, where there are
// fewer block rows than the device holds CTAs, to a cluster of up to 8 (its
// parts, hcsr_split); each CTA's R partial sums live in its shared memory (or,
// for block rows too tall for it, in a global scratch slice of its own).
// In the row-range phase every row belongs to one of the block row's warps: of
// W warps, warp w owns rows [ceil(w*rows/W), ceil((w+1)*rows/W)); in the COO
// phase the warps of a CTA add in turn.  The summation order of every row is
// therefore fixed and the result bitwise reproducible run to run (no float
// atomics).
//
// The block columns are taken in windows of kHWin blocks: the window's
// non-empty blocks are compacted into a row-range list and a COO list in
// shared memory (so the metadata staged never depends on b_n), then
//   * row-range phase: each warp walks, in block order, every CSR block and
//     every COO block of at least kHBig nonzeros for its own rows.  A CSR
//     block's nonzeros of those rows are one contiguous range, streamed in
//     chunks of 256 (8 consecutive nonzeros per lane, 16-byte loads of values
//     and uint16 columns); the rows starting inside a chunk are marked from
//     the block's row_ptr (a window of 32 row starts per lane set, loaded one
//     window ahead), each lane sums its 8 products split at the marks, and a
//     reverse segmented warp scan closes the rows that cross lanes, so each
//     row piece of a chunk is added to the accumulator exactly once.  A large
//     COO block keeps its nonzeros in row order (the builder writes them so):
//     the warp finds its range by a 32-ary search on the rows and streams it
//     the same way, a row starting wherever the row changes; a CTA that finds
//     rows out of order there starts its block row over with every COO block
//     in the COO phase;
//   * COO phase: the window's other COO nonzeros (in block order; a cluster's
//     CTAs take consecutive shares of them) are cut into rounds of 512; warp w
//     takes the w-th 64 of a round, 32 at a time (the block of each nonzero
//     from the compacted list: a warp-wide OR of the next block starts and a
//     popcount).  A run of one row inside one block is summed first, by a
//     segmented warp scan; lanes that hold the same row are ranked by a warp
//     match.  Then the warp waits for its turn, adds its sums into the rows,
//     rank by rank, and hands the turn on through a named barrier, so that
//     every row receives its sums in stream order.  Only the adds lie inside
//     the turn: loads, gathers, products and ranks of the other warps go on
//     meanwhile.
// A COO row index at or beyond the block row's rows (malformed input; the
// builder never writes one) is skipped rather than written out of range.
// Per row and part, the sum is: row-range pieces of window 0 in block order,
// COO sums of window 0 in stream order, then window 1, ...; the parts are added
// in order, and y = alpha*sum + beta*y (y is not read when beta == 0).
//
// What bounds it: the latency of the chain list -> row/column -> x in both
// phases, at 32 warps per SM (issue slots 43 % busy, LSU 56 %, DRAM 17 % on the
// power law of 1M rows, 19.6M nonzeros, R = C = 2000, fp64).  COO products
// that went through shared memory to the warp that owns their row, which
// filtered them out of each round, cost 350 instructions per 32 nonzeros and a
// barrier per round, with 16-warp CTAs: 223 us; in turns 149, and 141 with the
// carveout at the size the CTAs need (uniformly random columns 447 -> 244, the
// power law of 2M rows 454 -> 294, stencil 100^3, all CSR blocks, 129 -> 110).
// A turn of 32 nonzeros takes 162 us for the first, one of 128 149 (64: 149).
// Shared memory is sized for four CTAs per SM and the carveout asks for no
// more, so that the rest of the SM's 256 KB serves as L1 for the gathers of x.
//
// Mixed forms: lane sums of the CSR phase in compensated fp32 (two-sum), COO
// products in fp32; the block-row accumulator, where pieces of different
// blocks meet, is fp64.
#include <algorithm>
#include <cstring>
#include <string>
#include <type_traits>

#include "crs_merge.cuh"
#include "crs_run.cuh"
#include "hcsr_share.h"
#include "rvvla_internal.cuh"

namespace rvvla {
namespace {

constexpr uint32_t kHKindMask = 0x3FFFFFFFu;
constexpr int kHW = 8;                     // warps per CTA
constexpr int kHT = 32 * kHW;              // threads per CTA
constexpr int kHMinBlocks = 4;             // resident CTAs per SM the registers are sized for
constexpr int kHPer = 1;                   // block columns per thread in a window
constexpr int kHWin = kHPer * kHT;         // block columns per window
constexpr int kHProbe = kHWin / 32;        // list entries between the first probes of a search
static_assert(kHProbe >= 1 && kHProbe <= 32, "two steps of 32 probes reach every list entry");
constexpr int kHU = 2;                     // sub-steps of 32 COO nonzeros in a warp's turn
constexpr int kHRound = kHW * kHU * 32;    // COO nonzeros of one turn of every warp
static_assert(kHW <= 15, "one named barrier per warp beside barrier 0");
constexpr int kHBig = 1024;                // COO blocks of at least this many nonzeros take the row-range path
constexpr int kHLane = 8;                  // CSR nonzeros per lane and chunk
constexpr int kHChunk = 32 * kHLane;

// a non-empty block of the window: COO stream start (COO list only), nonzero
// offset, row_ptr offset, block column
struct HBlk {
  int cs;
  int bp;
  uint32_t off;
  int j;
};
static_assert(sizeof(HBlk) == 16, "HBlk is one 16-byte shared-memory load");

__host__ __device__ constexpr size_t hal16(size_t b) { return (b + 15) / 16 * 16; }

// Dynamic shared memory: [acc] list | per-warp row marks | per-warp mark groups.
template <class SA>
struct HLayout {
  size_t acc, list, mark, mgrp, total;
  __host__ __device__ explicit HLayout(int64_t racc) {
    acc = 0;
    list = hal16((size_t)racc * sizeof(SA));
    mark = list + hal16((size_t)(kHWin + 1) * sizeof(HBlk));
    mgrp = mark + (size_t)kHW * kHChunk * 4;
    total = mgrp + (size_t)kHW * 32 * 4;
  }
};

template <class V, class X, class SA, bool MIX>
struct HTypes {
  using Ac = std::conditional_t<MIX, CompF32, SA>;  // CSR lane sums
  using P = SA;                                     // a COO run sum (fp64 in the mixed forms)
  using PT = decltype(vmul(V(), X()));              // a product
};

// The turns of the warps: a warp waits on its own barrier for the warp before
// it, and hands on by arriving at the next warp's.
__device__ __forceinline__ void hcsr_turn_wait(int warp) {
  asm volatile("barrier.cta.sync %0, 64;" ::"r"(1 + warp) : "memory");
}
__device__ __forceinline__ void hcsr_turn_pass(int warp) {
  asm volatile("barrier.cta.arrive %0, 64;" ::"r"(1 + (warp + 1) % kHW) : "memory");
}

// Exclusive CTA-wide scan of three counters; t* are the CTA totals.
__device__ __forceinline__ void hcsr_scan3(int a, int b, int c, int& pa, int& pb, int& pc, int& ta, int& tb,
                                           int& tc, int* s_w) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int ia = a, ib = b, ic = c;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int oa = __shfl_up_sync(0xffffffffu, ia, d);
    const int ob = __shfl_up_sync(0xffffffffu, ib, d);
    const int oc = __shfl_up_sync(0xffffffffu, ic, d);
    if (lane >= d) {
      ia += oa;
      ib += ob;
      ic += oc;
    }
  }
  if (lane == 31) {
    s_w[warp] = ia;
    s_w[kHW + warp] = ib;
    s_w[2 * kHW + warp] = ic;
  }
  __syncthreads();
  int wa = 0, wb = 0, wc = 0;
  ta = tb = tc = 0;
#pragma unroll
  for (int w = 0; w < kHW; ++w) {
    const int va = s_w[w], vb = s_w[kHW + w], vc = s_w[2 * kHW + w];
    if (w < warp) {
      wa += va;
      wb += vb;
      wc += vc;
    }
    ta += va;
    tb += vb;
    tc += vc;
  }
  pa = wa + ia - a;
  pb = wb + ib - b;
  pc = wc + ic - c;
  __syncthreads();
}

// kHLane uint16 columns with 16-byte loads
__device__ __forceinline__ void hcsr_cols(const uint16_t* p, uint32_t (&c)[kHLane], uint64_t pol) {
#pragma unroll
  for (int h = 0; h < kHLane / 8; ++h) {
    const int4 t = ld_v4_l1(p + 8 * h, pol);
    const uint32_t w[4] = {(uint32_t)t.x, (uint32_t)t.y, (uint32_t)t.z, (uint32_t)t.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      c[8 * h + 2 * q] = w[q] & 0xFFFFu;
      c[8 * h + 2 * q + 1] = w[q] >> 16;
    }
  }
}

// kHLane values with 16-byte loads
template <class V>
__device__ __forceinline__ void hcsr_vals(const V* p, V (&v)[kHLane], uint64_t pol) {
  constexpr int E = 16 / (int)sizeof(V);  // values per load
#pragma unroll
  for (int q = 0; q < kHLane / E; ++q) {
    const int4 t = ld_v4_l1(p + E * q, pol);
    V tmp[E];
    static_assert(sizeof(tmp) == sizeof(int4), "one 16-byte load");
    memcpy(tmp, &t, sizeof(int4));
#pragma unroll
    for (int e = 0; e < E; ++e) v[E * q + e] = tmp[e];
  }
}

template <class V>
__device__ __forceinline__ V hcsr_ld1(const V* p) {
  if constexpr (std::is_same_v<V, __nv_bfloat16>) return __ushort_as_bfloat16(__ldg((const unsigned short*)p));
  else return __ldg(p);
}

template <class SA, class T>
__device__ __forceinline__ void hcsr_add(SA* acc, int r, T v) {
  acc[r] += (SA)v;
}

// Row-range phase of one warp for one CSR block: the nonzeros of the warp's
// rows [ra, rb).  Chunks of kHChunk nonzeros, kHLane consecutive ones per
// lane (16-byte loads): positions count from the block's first nonzero
// rounded down to a multiple of 8, so a chunk start is 16-byte aligned
// whenever the arrays are (VEC).  Row starts come from the block's row_ptr
// in windows of 32 rows (the next window loaded one window ahead) and mark
// the lanes' slots through a per-warp table; each lane sums its products
// split at the marks, and a reverse segmented scan adds the parts of rows
// crossing lanes.  When no lane holds two row starts (rows of 8 or more
// nonzeros), a lane's sums take the short split at its one mark.  The
// columns of a chunk are loaded one chunk ahead, so that its x gathers leave
// together with its value loads.
template <class V, class X, class SA, bool MIX, bool VEC>
__device__ __forceinline__ void hcsr_csr_rows(const uint32_t* __restrict__ rp, int64_t bp, int ra, int rb, int64_t nz,
                                              const uint16_t* __restrict__ col_idx, const V* __restrict__ values,
                                              const X* __restrict__ xb, SA* acc, int* table, uint32_t* mgrp, int lane,
                                              uint64_t pf, uint64_t pl) {
  using Ty = HTypes<V, X, SA, MIX>;
  using Ac = typename Ty::Ac;
  using PT = typename Ty::PT;
  using CT = SA;
  const int64_t base = bp & ~(int64_t)7;
  const uint32_t off = (uint32_t)(bp - base);
  const uint32_t lo = off + __ldg(rp + ra), hi = off + __ldg(rp + rb);
  if (lo >= hi) return;
  const uint32_t lim = (uint32_t)(nz - base);  // positions below lim lie inside the arrays
  const V* __restrict__ vb = values + base;
  const uint16_t* __restrict__ cb = col_idx + base;
  int wb = ra;
  auto ldwin = [&](int b0, uint32_t& s, uint32_t& e) {
    const int r = b0 + lane;
    s = r < rb ? off + __ldg(rp + r) : 0xFFFFFFFFu;
    e = r < rb ? off + __ldg(rp + r + 1) : 0xFFFFFFFFu;
  };
  uint32_t s_c, e_c, s_n, e_n;
  ldwin(wb, s_c, e_c);
  ldwin(wb + 32, s_n, e_n);
  int open_row = -1;
  // the lane's 8 columns of the next chunk, loaded one chunk ahead, so that
  // a chunk's x gathers leave together with its value loads
  const uint32_t c0 = lo & ~7u;
  int4 cn = make_int4(0, 0, 0, 0);
  if (VEC && c0 + kHLane * lane + kHLane <= lim) cn = ld_v4_l1(cb + c0 + kHLane * lane, pf);
  for (uint32_t c = c0; c < hi; c += kHChunk) {
    const uint32_t a = c + kHLane * lane;
    const uint32_t fv = lo > a ? lo - a : 0u;  // the lane's slots in [fv, lv) lie in [lo, hi)
    const uint32_t lv = hi > a ? hi - a : 0u;
    const int4 cw = cn;
    if (VEC) {
      const uint32_t an = a + kHChunk;
      cn = c + kHChunk < hi && an + kHLane <= lim ? ld_v4_l1(cb + an, pf) : make_int4(0, 0, 0, 0);
    }
    // ---- loads and products
    PT p[kHLane];
    {
      V vv[kHLane];
      uint32_t cc[kHLane];
      if (VEC && a + kHLane <= lim) {
        hcsr_vals(vb + a, vv, pf);
        const uint32_t w[4] = {(uint32_t)cw.x, (uint32_t)cw.y, (uint32_t)cw.z, (uint32_t)cw.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          cc[2 * q] = w[q] & 0xFFFFu;
          cc[2 * q + 1] = w[q] >> 16;
        }
      } else {
#pragma unroll
        for (int i = 0; i < kHLane; ++i) {
          const bool in = a + i < lim;
          vv[i] = in ? hcsr_ld1(vb + a + i) : V(0);
          cc[i] = in ? (uint32_t)__ldg(cb + a + i) : 0u;
        }
      }
#pragma unroll
      for (int i = 0; i < kHLane; ++i) {
        const bool ok = (uint32_t)i >= fv && (uint32_t)i < lv;
        if constexpr (MIX) p[i] = ok ? to_f32(vv[i]) * (float)ld_keep(xb + cc[i], pl) : 0.f;
        else p[i] = ok ? vv[i] * ld_keep(xb + cc[i], pl) : PT(0);
      }
    }
    // ---- marks of the rows that start inside the chunk
    mgrp[lane] = 0u;
    __syncwarp();
    for (;;) {
      const uint32_t pos = s_c - c;  // wraps for rows that started before the chunk
      if (pos < (uint32_t)kHChunk && s_c < e_c) {
        table[pos] = wb + lane;
        atomicOr(mgrp + pos / kHLane, 1u << (pos % kHLane));
      }
      const uint32_t s31 = __shfl_sync(0xffffffffu, s_c, 31);
      if (!(wb + 32 < rb && s31 < c + kHChunk)) break;
      wb += 32;
      s_c = s_n;
      e_c = e_n;
      ldwin(wb + 32, s_n, e_n);
    }
    __syncwarp();
    const uint32_t mb = mgrp[lane];
    // ---- lane sums: lead = before the lane's first mark, sum = from its last
    // mark; rows that start and end inside the lane are added now
    Ac sum, lead;
    acc_zero(sum);
    acc_zero(lead);
    int nf = 0, rcur = -1;
    if (!__any_sync(0xffffffffu, (mb & (mb - 1u)) != 0u)) {
      const int m = mb ? __ffs(mb) - 1 : kHLane;
#pragma unroll
      for (int i = 0; i < kHLane; ++i) {
        if (i == m) {
          lead = sum;
          acc_zero(sum);
        }
        acc_add(sum, p[i]);
      }
      if (mb) {
        nf = 1;
        rcur = table[kHLane * lane + m];
      } else {
        lead = sum;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kHLane; ++i) {
        if ((mb >> i) & 1u) {
          if (nf == 0) lead = sum;
          else hcsr_add(acc, rcur, acc_carry(sum));
          rcur = table[kHLane * lane + i];
          ++nf;
          acc_zero(sum);
        }
        acc_add(sum, p[i]);
      }
      if (nf == 0) lead = sum;
    }
    // ---- rows crossing lanes: reverse segmented scan of the leads
    const unsigned marks = __ballot_sync(0xffffffffu, nf > 0);
    const unsigned ge = marks & (~0u << lane);
    const int e = ge ? __ffs(ge) - 1 : 31;
    CT T = (CT)acc_carry(lead);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const CT o = __shfl_down_sync(0xffffffffu, T, d);
      if (lane + d <= e) T += o;
    }
    CT Tn = __shfl_down_sync(0xffffffffu, T, 1);
    if (lane == 31) Tn = CT(0);
    const CT T0 = __shfl_sync(0xffffffffu, T, 0);
    if (lane == 0 && open_row >= 0) hcsr_add(acc, open_row, T0);
    if (nf > 0) hcsr_add(acc, rcur, (CT)acc_carry(sum) + Tn);
    if (marks) open_row = __shfl_sync(0xffffffffu, rcur, 31 - __clz(marks));
    __syncwarp();
  }
}

// First k in [0, cnt) with rows[k] >= t (cnt when none), for ascending rows;
// a 32-ary search of the warp (each step probes 32 positions).  On rows that
// do not ascend the result is some k in [0, cnt].
__device__ __forceinline__ int hcsr_lower_bound(const uint32_t* __restrict__ rows, int cnt, uint32_t t, int lane) {
  int lo = 0, hi = cnt;  // the answer lies in [lo, hi]
  while (hi - lo > 32) {
    const int k = lo + (int)(((int64_t)(hi - lo) * lane) >> 5);
    const int c = __popc(__ballot_sync(0xffffffffu, __ldg(rows + k) < t));
    const int nlo = c > 0 ? __shfl_sync(0xffffffffu, k, (c - 1) & 31) + 1 : lo;
    const int nhi = c < 32 ? __shfl_sync(0xffffffffu, k, c & 31) : hi;
    lo = nlo;
    hi = max(nhi, nlo);
  }
  const bool less = lo + lane < hi && __ldg(rows + lo + lane) < t;
  return lo + __popc(__ballot_sync(0xffffffffu, less));
}

// Row-range phase of one warp for one large COO block: the nonzeros
// [lo, hi) (absolute) that hold the warp's rows [ra, rb), in chunks of 256 as
// in hcsr_csr_rows.  rp holds each nonzero's row (rp[k - bp]); a row starts
// where the row differs from the previous kept nonzero's.  Returns true when
// a row descends or lies outside [ra, rb); such nonzeros are left out.
template <class V, class X, class SA, bool MIX, bool VEC>
__device__ __forceinline__ bool hcsr_coo_rows(const uint32_t* __restrict__ rp, int64_t bp, int ra, int rb, int64_t lo,
                                              int64_t hi, int64_t nz, const uint16_t* __restrict__ col_idx,
                                              const V* __restrict__ values, const X* __restrict__ xb, SA* acc,
                                              int lane, uint64_t pf, uint64_t pl) {
  using Ty = HTypes<V, X, SA, MIX>;
  using Ac = typename Ty::Ac;
  using PT = typename Ty::PT;
  using CT = SA;
  uint32_t last_row = 0xFFFFFFFFu;   // row of the last nonzero before the chunk
  uint32_t last_kept = 0xFFFFFFFFu;  // the same, of the kept nonzeros
  bool bad = false;
  int open_row = -1;
  for (int64_t c = lo & ~(int64_t)7; c < hi; c += kHChunk) {
    const int64_t a = c + kHLane * lane;
    // ---- rows (0xFFFFFFFF outside [lo, hi) and outside [ra, rb))
    uint32_t rw[kHLane];
    {
#pragma unroll
      for (int i = 0; i < kHLane; ++i) rw[i] = a + i >= lo && a + i < hi ? __ldg(rp + (a + i - bp)) : 0xFFFFFFFFu;
      uint32_t before = __shfl_up_sync(0xffffffffu, rw[kHLane - 1], 1);
      if (lane == 0) before = last_row;
      const uint32_t l31 = __shfl_sync(0xffffffffu, rw[kHLane - 1], 31);
      last_row = l31 != 0xFFFFFFFFu ? l31 : last_row;
#pragma unroll
      for (int i = 0; i < kHLane; ++i) {
        if (rw[i] != 0xFFFFFFFFu) {
          if ((before != 0xFFFFFFFFu && rw[i] < before) || rw[i] < (uint32_t)ra || rw[i] >= (uint32_t)rb) bad = true;
          before = rw[i];
          if (rw[i] < (uint32_t)ra || rw[i] >= (uint32_t)rb) rw[i] = 0xFFFFFFFFu;
        }
      }
    }
    // ---- loads and products
    PT p[kHLane];
    {
      V vv[kHLane];
      uint32_t cc[kHLane];
      const bool any = a < hi && a + kHLane > lo;
      if (VEC && any && a + kHLane <= nz) {
        hcsr_vals(values + a, vv, pf);
        hcsr_cols(col_idx + a, cc, pf);
      } else {
#pragma unroll
        for (int i = 0; i < kHLane; ++i) {
          const bool ok = a + i >= lo && a + i < hi;
          vv[i] = ok ? hcsr_ld1(values + a + i) : V(0);
          cc[i] = ok ? (uint32_t)__ldg(col_idx + a + i) : 0u;
        }
      }
#pragma unroll
      for (int i = 0; i < kHLane; ++i) {
        const bool ok = rw[i] != 0xFFFFFFFFu;
        if constexpr (MIX) p[i] = ok ? to_f32(vv[i]) * (float)ld_keep(xb + cc[i], pl) : 0.f;
        else p[i] = ok ? vv[i] * ld_keep(xb + cc[i], pl) : PT(0);
      }
    }
    // ---- marks of the rows that start inside the chunk
    uint32_t mb = 0;
    {
      // a row starts where it differs from the previous kept nonzero's
      uint32_t prev = __shfl_up_sync(0xffffffffu, rw[kHLane - 1], 1);
      if (lane == 0) prev = last_kept;
#pragma unroll
      for (int i = 0; i < kHLane; ++i) {
        const uint32_t before = i == 0 ? prev : rw[i - 1];
        if (rw[i] != 0xFFFFFFFFu && rw[i] != before) mb |= 1u << i;
      }
      const uint32_t k31 = __shfl_sync(0xffffffffu, rw[kHLane - 1], 31);
      last_kept = k31 != 0xFFFFFFFFu ? k31 : last_kept;
    }
    // ---- lane sums split at the marks; rows closed inside the lane are added now
    Ac sum, lead;
    acc_zero(sum);
    acc_zero(lead);
    int nf = 0, rcur = -1;
#pragma unroll
    for (int i = 0; i < kHLane; ++i) {
      if ((mb >> i) & 1u) {
        if (nf == 0) lead = sum;
        else hcsr_add(acc, rcur, acc_carry(sum));
        rcur = (int)rw[i];
        ++nf;
        acc_zero(sum);
      }
      acc_add(sum, p[i]);
    }
    if (nf == 0) lead = sum;
    // ---- rows crossing lanes: reverse segmented scan of the leads
    const unsigned marks = __ballot_sync(0xffffffffu, nf > 0);
    const unsigned ge = marks & (~0u << lane);
    const int e = ge ? __ffs(ge) - 1 : 31;
    CT T = (CT)acc_carry(lead);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const CT o = __shfl_down_sync(0xffffffffu, T, d);
      if (lane + d <= e) T += o;
    }
    CT Tn = __shfl_down_sync(0xffffffffu, T, 1);
    if (lane == 31) Tn = CT(0);
    const CT T0 = __shfl_sync(0xffffffffu, T, 0);
    if (lane == 0 && open_row >= 0) hcsr_add(acc, open_row, T0);
    if (nf > 0) hcsr_add(acc, rcur, (CT)acc_carry(sum) + Tn);
    if (marks) open_row = __shfl_sync(0xffffffffu, rcur, 31 - __clz(marks));
    __syncwarp();
  }
  return bad;
}

// Barrier of the CTAs that share a block row; shared memory written before it
// is visible to them after it.
__device__ __forceinline__ void hcsr_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The shared-memory address of p in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t hcsr_peer(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void hcsr_peer_ld(uint32_t a, int& v) {
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void hcsr_peer_ld(uint32_t a, float& v) {
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void hcsr_peer_ld(uint32_t a, double& v) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}

// Raw loads of one COO sub-step (32 consecutive COO nonzeros of the window).
template <class V>
struct HCooRaw {
  uint32_t row;
  uint32_t col;
  V v;
  int64_t xoff;
  bool ok;
};

template <class V, class X, class SA, bool MIX, bool VEC, bool GACC, bool SPLIT>
__global__ void __launch_bounds__(kHT, kHMinBlocks)
hcsr_spmv_kernel(int64_t R, int64_t C, int64_t m, int64_t nz, int64_t b_n, const int* __restrict__ block_ptr,
                 const uint32_t* __restrict__ row_offset, const uint32_t* __restrict__ row_ptr,
                 const uint16_t* __restrict__ col_idx, const V* __restrict__ values, const X* __restrict__ x,
                 X* __restrict__ y, X alpha, X beta, SA* __restrict__ gacc, int parts) {
  using Ty = HTypes<V, X, SA, MIX>;
  using P = typename Ty::P;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_w[3 * kHW];
  const HLayout<SA> L(GACC ? 0 : min(R, m));  // as the launch sizes it
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int split = SPLIT ? parts : 1;  // CTAs (one cluster) that share a block row
  const int64_t br = blockIdx.x / (unsigned)split;
  const int part = (int)(blockIdx.x % (unsigned)split);
  const int64_t r0 = br * R;
  const int rows = (int)min(R, m - r0);
  SA* acc = GACC ? gacc + part * m + r0 : reinterpret_cast<SA*>(smem + L.acc);
  HBlk* list = reinterpret_cast<HBlk*>(smem + L.list);
  int* table = reinterpret_cast<int*>(smem + L.mark) + warp * kHChunk;
  uint32_t* mgrp = reinterpret_cast<uint32_t*>(smem + L.mgrp) + warp * 32;
  __shared__ int s_bad;  // a large COO block whose rows do not ascend was met
  bool big_ok = true;
  const uint64_t pf = policy_evict_first(), pl = policy_evict_last();

  for (int li = tid; li < rows; li += kHT) acc[li] = SA(0);
  if (tid == 0) s_bad = 0;
  // this warp's rows
  const int owner = part * kHW + warp, owners = split * kHW;
  const int ra = (int)(((int64_t)owner * rows + owners - 1) / owners);
  const int rb = (int)(((int64_t)(owner + 1) * rows + owners - 1) / owners);
  const int64_t blk0 = br * b_n;
  __syncthreads();

  for (;;) {
  for (int64_t jw = 0; jw < b_n; jw += kHWin) {
    const int nb = (int)(b_n - jw < kHWin ? b_n - jw : kHWin);
    // ---- compact the window's non-empty blocks (kHPer consecutive per thread):
    // CSR blocks and COO blocks of >= kHBig nonzeros form the row-range list
    // (block order, from the back of `list`), the smaller COO blocks the COO
    // stream (from the front, with a sentinel)
    int bpq[kHPer], cntq[kHPer];
    uint32_t roq[kHPer];
    int kindq[kHPer];  // 0 none, 1 CSR, 2 large COO, 3 small COO
#pragma unroll
    for (int q = 0; q < kHPer; ++q) {
      const int jj = kHPer * tid + q;
      bpq[q] = 0;
      cntq[q] = 0;
      roq[q] = 0u;
      kindq[q] = 0;
      if (jj < nb) {
        const int64_t b = blk0 + jw + jj;
        bpq[q] = block_ptr[b];
        cntq[q] = block_ptr[b + 1] - bpq[q];
        roq[q] = row_offset[b];
        if (cntq[q] > 0) kindq[q] = (roq[q] >> 30) == 1u ? 1 : (cntq[q] >= kHBig && big_ok ? 2 : 3);
      }
    }
    int n_seg = 0, n_coo = 0, n_ent = 0;
#pragma unroll
    for (int q = 0; q < kHPer; ++q) {
      if (kindq[q] == 1 || kindq[q] == 2) ++n_seg;
      if (kindq[q] == 3) {
        ++n_coo;
        n_ent += cntq[q];
      }
    }
    int p_seg, p_coo, p_ent, t_seg, t_coo, t_ent;
    hcsr_scan3(n_seg, n_coo, n_ent, p_seg, p_coo, p_ent, t_seg, t_coo, t_ent, s_w);
#pragma unroll
    for (int q = 0; q < kHPer; ++q) {
      if (kindq[q] == 0) continue;
      HBlk h;
      h.bp = bpq[q];
      h.off = roq[q] & kHKindMask;
      h.j = (int)(jw + kHPer * tid + q);
      if (kindq[q] == 1 || kindq[q] == 2) {
        h.cs = kindq[q] == 1 ? -1 : cntq[q];  // a large COO block keeps its nonzero count
        list[kHWin + 1 - t_seg + p_seg++] = h;
      } else {
        h.cs = p_ent;
        p_ent += cntq[q];
        list[p_coo++] = h;
      }
    }
    if (tid == 0) list[t_coo].cs = t_ent;  // sentinel: end of the COO stream
    __syncthreads();

    // ---- row-range phase: this warp's rows of every CSR block and large
    // COO block of the window, in block order.  A large COO block's rows
    // ascend (the builder writes them so): the warp finds its nonzeros
    // [first row >= ra, first row >= rb) by search and checks, on the way,
    // that they ascend and lie in [ra, rb); a CTA whose warps met anything
    // else redoes its block row with every COO block in the COO stream.
    for (int i = 0; i < t_seg; ++i) {
      const HBlk h = list[kHWin + 1 - t_seg + i];
      const uint32_t* rp = row_ptr + h.off;
      if (h.cs < 0) {
        if (ra >= rb) continue;
        hcsr_csr_rows<V, X, SA, MIX, VEC>(rp, h.bp, ra, rb, nz, col_idx, values, x + (int64_t)h.j * C, acc, table,
                                          mgrp, lane, pf, pl);
      } else {
        const int cnt = h.cs;
        const int klo = owner == 0 ? 0 : hcsr_lower_bound(rp, cnt, (uint32_t)ra, lane);
        const int khi = owner == owners - 1 ? cnt : hcsr_lower_bound(rp, cnt, (uint32_t)rb, lane);
        if (klo > khi) {
          if (lane == 0) s_bad = 1;
          continue;
        }
        if (klo == khi) continue;
        if (hcsr_coo_rows<V, X, SA, MIX, VEC>(rp, h.bp, ra, rb, (int64_t)h.bp + klo, (int64_t)h.bp + khi, nz, col_idx,
                                              values, x + (int64_t)h.j * C, acc, lane, pf, pl))
          s_bad = 1;
      }
    }

    // ---- COO phase: rounds of kHRound nonzeros of the window's COO stream
    // (this CTA's share: nonzeros [qs.lo, qs.hi) of it)
    const HcsrShare qs = hcsr_share(t_ent, split, part);
    if (qs.lo < qs.hi) {
      const int ncoo = t_coo;
      const unsigned ntot = (unsigned)qs.hi;
      const int nrounds = qs.rounds(kHRound);
      HCooRaw<V> raw[kHU];
      auto coo_load = [&](int t) {
        const unsigned q00 = qs.first(t, kHRound, warp * (kHU * 32));
        // the block of the warp's first nonzero: the last that starts at or
        // before it, by two steps of 32 probes (list[0].cs is 0)
        const int qa = (int)min(q00, ntot - 1u);
        int ia = lane * kHProbe < ncoo && list[lane * kHProbe].cs <= qa;
        ia = kHProbe * (__popc(__ballot_sync(0xffffffffu, ia)) - 1);
        const bool le = lane < kHProbe && ia + lane < ncoo && list[ia + lane].cs <= qa;
        ia += __popc(__ballot_sync(0xffffffffu, le)) - 1;
#pragma unroll
        for (int u = 0; u < kHU; ++u) {
          const unsigned q0 = q00 + 32u * u;
          const int nxt = ia + 1 + lane;
          const int d = nxt <= ncoo ? (int)((unsigned)list[nxt].cs - q0) : 32;
          const unsigned mask = __reduce_or_sync(0xffffffffu, (d >= 0 && d < 32) ? 1u << d : 0u);
          int blk = ia + __popc(mask & ((2u << lane) - 1u));
          blk = min(blk, ncoo - 1);
          const unsigned q = q0 + lane;
          HCooRaw<V>& r = raw[u];
          r.ok = q < ntot;
          r.row = 0u;
          r.xoff = -1;
          if (r.ok) {
            const HBlk h = list[blk];
            const int e = (int)q - h.cs;
            const int64_t k = (int64_t)h.bp + e;
            r.row = ld_stream(row_ptr + h.off + e, pf);
            r.col = (uint32_t)ld_stream(col_idx + k, pf);
            r.v = ld_stream(values + k, pf);
            r.xoff = (int64_t)h.j * C;
            r.ok = r.row < (uint32_t)rows;  // a row beyond the block row (malformed input) is skipped
          }
          ia = __shfl_sync(0xffffffffu, blk, 31);
        }
      };
      coo_load(0);
      __syncthreads();  // the row-range phase of every warp is over
      for (int t = 0; t < nrounds; ++t) {
        X xv[kHU];
#pragma unroll
        for (int u = 0; u < kHU; ++u) xv[u] = raw[u].ok ? ld_keep(x + raw[u].xoff + raw[u].col, pl) : X(0);
        uint32_t row[kHU];
        P pr[kHU];
        int rank[kHU], last[kHU];
#pragma unroll
        for (int u = 0; u < kHU; ++u) {
          const HCooRaw<V>& r = raw[u];
          P pv = P(0);
          if (r.ok) {
            if constexpr (MIX) pv = (P)(to_f32(r.v) * (float)xv[u]);
            else pv = (P)(r.v * xv[u]);
          }
          // runs of one row inside one block (consecutive lanes) are summed
          // here, into the run's last lane
          // (cont: this lane continues the previous lane's run; most
          // sub-steps have none, and skip the scan)
          const uint32_t prow = __shfl_up_sync(0xffffffffu, r.row, 1);
          const int64_t pxo = __shfl_up_sync(0xffffffffu, r.xoff, 1);
          const bool cont = lane > 0 && r.ok && prow == r.row && pxo == r.xoff;
          bool tail = r.ok;
          if (__any_sync(0xffffffffu, cont)) {
            pv = warp_seg_scan(pv, !cont, lane);
            const bool ncont = __shfl_down_sync(0xffffffffu, cont, 1);
            tail = r.ok && (lane == 31 || !ncont);
          }
          // lanes that hold the same row add one after another, in lane order
          row[u] = r.row;
          pr[u] = pv;
          const unsigned peers = __match_any_sync(0xffffffffu, tail ? row[u] : 0xFFFFFFFFu);
          rank[u] = tail ? __popc(peers & ((1u << lane) - 1u)) : -1;
          last[u] = __reduce_max_sync(0xffffffffu, rank[u]);
        }
        if (t + 1 < nrounds) coo_load(t + 1);
        // the warps take turns, so every row receives its sums in stream order
        if (t > 0 || warp > 0) hcsr_turn_wait(warp);
#pragma unroll
        for (int u = 0; u < kHU; ++u) {
          for (int k = 0; k <= last[u]; ++k) {
            if (rank[u] == k) acc[row[u]] += pr[u];
            __syncwarp();
          }
        }
        if (t + 1 < nrounds || warp + 1 < kHW) hcsr_turn_pass(warp);
      }
    }
    __syncthreads();
  }
  int bad = s_bad;
  if constexpr (SPLIT) {
    hcsr_cluster_sync();  // every CTA's sums of the block row are complete
    for (int k = 0; k < split; ++k) {
      int b;
      hcsr_peer_ld(hcsr_peer(&s_bad, k), b);
      bad |= b;
    }
  }
  if (!big_ok || !bad) break;
  // rows of a large COO block out of order: start over, all COO blocks
  // through the COO stream (the CTAs of a cluster together)
  big_ok = false;
  __syncthreads();
  for (int li = tid; li < rows; li += kHT) acc[li] = SA(0);
  __syncthreads();
  }
  // the CTAs' sums of a row are added in the order of the parts
  const int fa = (int)((int64_t)part * rows / split), fb = (int)((int64_t)(part + 1) * rows / split);
  for (int li = fa + tid; li < fb; li += kHT) {
    SA sum = SA(0);
    if constexpr (!SPLIT) {
      sum = acc[li];
    } else {
      for (int k = 0; k < split; ++k) {
        SA v;
        if constexpr (GACC) v = __ldcg(gacc + k * m + r0 + li);
        else hcsr_peer_ld(hcsr_peer(acc + li, k), v);
        sum += v;
      }
    }
    const X o = (X)sum;
    X* yp = y + r0 + li;
    *yp = (beta == X(0)) ? alpha * o : alpha * o + beta * *yp;
  }
  if constexpr (SPLIT) hcsr_cluster_sync();  // no CTA leaves while its sums are read
}

int hcsr_validate(const rvvla_hcsr* A, const void* x, const void* y) {
  if (!A) return fail(RVVLA_ERR_INVALID_ARG, "hcsr: null descriptor");
  if (A->R <= 0 || A->C <= 0 || A->m < 0 || A->n < 0 || A->nz < 0)
    return fail(RVVLA_ERR_INVALID_ARG, "hcsr: bad sizes");
  if (A->b_m != (A->m + A->R - 1) / A->R || A->b_n != (A->n + A->C - 1) / A->C)
    return fail(RVVLA_ERR_FORMAT, "hcsr: b_m/b_n inconsistent with m, n, R, C");
  if (A->m > 0 && (!A->block_ptr || !A->row_offset || !y)) return fail(RVVLA_ERR_INVALID_ARG, "hcsr: null array");
  if (A->nz > 0 && (!A->col_idx || !A->values || !A->row_ptr || !x))
    return fail(RVVLA_ERR_INVALID_ARG, "hcsr: null array");
  if (A->C > 65536) return fail(RVVLA_ERR_TOO_LARGE, "hcsr: C > 65536 does not fit the uint16 col_idx");
  if (A->m > INT32_MAX || A->nz > INT32_MAX) return fail(RVVLA_ERR_TOO_LARGE, "hcsr: m or nz beyond 2^31 - 1");
  return RVVLA_OK;
}

// Largest dynamic shared memory one CTA may take: 227 KB on sm_100a, less the
// static arrays.
constexpr size_t kHSmemMax = 226 * 1024;


// CTAs per block row: as many as keep all CTAs resident at once (cluster
// sizes need not be powers of two; an eighth of the slots is left free, since a
// cluster lies within a GPC: 113 block rows take 53 us in clusters of 5, 565
// of 592 slots, and 45 in clusters of 4).  Each part walks the block list and
// row pointers again, so more CTAs than that lose (1M rows in 501 block rows,
// measured with 16-warp CTAs, two per SM: 1, 2, 4 parts 191, 215, 279 us) and
// fewer leave SMs idle (power law, fp64, 100K rows in 50 block rows 67 -> 35
// us, 300K rows 93 -> 62, 30K rows 60 -> 27; fp32 with R = 4000, 1M rows in 251
// block rows 166 -> 117; accumulators in scratch, 1M rows, R = 60000, fp64
// 2317 -> 477).  Blocks that take the row-range path (large ones) are searched by
// every warp of the block row, so where the average block is one, a warp's share
// of it is kept at kHSplitBlk nonzeros (hcsr_parts).  Random rows, parts by that
// rule / by the slots alone / 16-warp CTAs without parts: fp32 n = 357K mean 39
// 370 / 510 / 367 us (2 and 5 parts), 200K mean 30 193 / 285 / 193 (3, 8), 500K
// mean 40 502 / 702 / 517 (1, 4); fp64 100K mean 40 205 / 314 / 203 (2, 8), 150K
// mean 40 333 / 451 / 312 (1, 6).  64 and 128 nonzeros: 366 and 425, 195 and 180,
// 513 and 502, 222 and 190, 331 and 334.
int hcsr_split(const rvvla_hcsr* A, size_t smem) {
  const int64_t per_sm = std::min<int64_t>(kHMinBlocks, (kHSmemMax + 2048) / (smem + 2048));
  return hcsr_parts(A->b_m, A->b_n, A->nz, sm_count() * per_sm * 7 / 8, kHW, kHBig);
}

template <class V, class X, class SA, bool MIX, bool VEC, bool GACC, bool SPLIT>
int hcsr_launch(const rvvla_hcsr* A, int split, X alpha, const X* x, X beta, X* y, SA* gacc, size_t smem, cudaStream_t st) {
  auto kern = hcsr_spmv_kernel<V, X, SA, MIX, VEC, GACC, SPLIT>;
  // the kernel's limit is common to all threads that launch it: always the
  // largest, not this call's, which another thread's smaller one could replace
  // before the launch
  RVVLA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHSmemMax));
  // shared memory for kHMinBlocks CTAs (1 KB of each is the system's), the
  // rest of the SM's 256 KB as L1: the gathers of x hit there.  The SM takes
  // one of a few sizes, and a wish above one of them gets the next.
  const size_t need = kHMinBlocks * (smem + 2048);
  int carve = 100;
  for (const int kb : {196, 164, 132, 100, 64})
    if (need <= (size_t)kb * 1024) carve = kb * 100 / 228;
  RVVLA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, carve));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(A->b_m * split));
  cfg.blockDim = dim3(kHT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim = {(unsigned)split, 1, 1};
  cfg.attrs = &at;
  cfg.numAttrs = SPLIT ? 1 : 0;
  RVVLA_CUDA(cudaLaunchKernelEx(&cfg, kern, A->R, A->C, A->m, A->nz, A->b_n, (const int*)A->block_ptr,
                                (const uint32_t*)A->row_offset, (const uint32_t*)A->row_ptr,
                                (const uint16_t*)A->col_idx, (const V*)A->values, x, y, alpha, beta, gacc, split));
  RVVLA_LAUNCHED("hcsr_spmv_kernel");
  return RVVLA_OK;
}

template <class V, class X, class SA, bool MIX>
int hcsr_spmv_impl(const rvvla_hcsr* A, X alpha, const X* x, X beta, X* y, cudaStream_t st) {
  int rc = hcsr_validate(A, x, y);
  if (rc) return rc;
  if (A->m == 0) return RVVLA_OK;
  if (A->b_m > INT32_MAX) return fail(RVVLA_ERR_TOO_LARGE, "hcsr: more than 2^31 - 1 block rows");
  const bool vec = ((uintptr_t)A->values % 16 == 0) && ((uintptr_t)A->col_idx % 16 == 0);
  const int64_t racc = std::min<int64_t>(A->R, A->m);
  const size_t smem_s = HLayout<SA>(racc).total;
  if (smem_s <= kHSmemMax) {
    const int split = hcsr_split(A, smem_s);
    if (split > 1)
      return vec ? hcsr_launch<V, X, SA, MIX, true, false, true>(A, split, alpha, x, beta, y, nullptr, smem_s, st)
                 : hcsr_launch<V, X, SA, MIX, false, false, true>(A, split, alpha, x, beta, y, nullptr, smem_s, st);
    return vec ? hcsr_launch<V, X, SA, MIX, true, false, false>(A, 1, alpha, x, beta, y, nullptr, smem_s, st)
               : hcsr_launch<V, X, SA, MIX, false, false, false>(A, 1, alpha, x, beta, y, nullptr, smem_s, st);
  }
  // block rows too tall for shared memory: the accumulators are a global
  // scratch array (each CTA owns its slice)
  const size_t smem_g = HLayout<SA>(0).total;
  int split = hcsr_split(A, smem_g);
  Scratch sc;
  cudaError_t e = sc.alloc_kept((size_t)split * A->m * sizeof(SA), st);
  if (e == cudaErrorMemoryAllocation && split > 1) {  // no room for a slice per part: one part
    cudaGetLastError();
    split = 1;
    e = sc.alloc_kept((size_t)A->m * sizeof(SA), st);
  }
  RVVLA_CUDA(e);
  return vec ? hcsr_launch<V, X, SA, MIX, true, true, true>(A, split, alpha, x, beta, y, sc.as<SA>(), smem_g, st)
             : hcsr_launch<V, X, SA, MIX, false, true, true>(A, split, alpha, x, beta, y, sc.as<SA>(), smem_g, st);
}

}  // namespace
}  // namespace rvvla

using namespace rvvla;

extern "C" {

int rvvla_hcsr_spmv_f64(const rvvla_hcsr* A, double alpha, const double* x, double beta, double* y, void* stream) {
  return hcsr_spmv_impl<double, double, double, false>(A, alpha, x, beta, y, as_stream(stream));
}

int rvvla_hcsr_spmv_f32(const rvvla_hcsr* A, float alpha, const float* x, float beta, float* y, void* stream) {
  return hcsr_spmv_impl<float, float, float, false>(A, alpha, x, beta, y, as_stream(stream));
}

int rvvla_hcsr_spmv_mixed(const rvvla_hcsr* A, int val_type, float alpha, const float* x, float beta, float* y,
                          void* stream) {
  if (val_type == RVVLA_F32)
    return hcsr_spmv_impl<float, float, double, true>(A, alpha, x, beta, y, as_stream(stream));
  if (val_type == RVVLA_BF16)
    return hcsr_spmv_impl<__nv_bfloat16, float, double, true>(A, alpha, x, beta, y, as_stream(stream));
  return fail(RVVLA_ERR_INVALID_ARG, "hcsr_spmv_mixed: val_type must be RVVLA_F32 or RVVLA_BF16");
}

}  // extern "C"
