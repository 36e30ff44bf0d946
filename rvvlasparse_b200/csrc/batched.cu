// batched.cu — many independent SpMVs (Y_i = alpha * A_i X_i + beta * Y_i,
// each X_i / Y_i holding k right-hand sides) in one call, with a CUDA-graph
// wrapper and a measuring autotuner.  No reference counterpart.
//
// Plan (rvvla_batched_plan): each matrix runs either as CSR (the caller's
// arrays) or as SELL-C-sigma (C = 32, built on the GPU and owned by the
// plan).  All CSR matrices are one launch over a list of tiles of
// bounded work, all SELL matrices another over shares of slices; a plan of one
// layout is one launch.
//
// Vectors: X_i is n_i x k and Y_i is m_i x k, row-major (the k values of one
// row contiguous), packed one matrix after another; x_off/y_off give each
// matrix's first element.  A nonzero (j, c) of row r needs the k contiguous
// values X[c*k .. c*k+k-1]: for k > 1, G = k * sizeof(T) / 16 lanes take 16
// bytes each (scalars when X or Y is not 16-byte aligned).
//
// What bounds it: the gathers of X rows.  From L2 they come at one 32-byte
// sector per clock and SM at best (290 G/s measured, whatever the size up to
// 64 MB; a 128-byte row takes 1.8 clocks), from L1 at three per clock, while
// HBM brings 2.8 fp32 nonzeros per clock and SM.
//
// SELL kernels: one CTA per SM, a contiguous share of the slices per CTA, so
// that all warps of an SM work on one matrix and its X rows stay in that SM's
// L1 (k = 1: 240 us with one CTA of 32 warps per SM, 340 with two of 16 on
// two shares, 410 with six of 8; a window of X in shared memory left L1 too
// few lines for the loads in flight, 301).  For rows of 32 bytes and more X
// does not fit L1 and balance counts more: each CTA takes four shorter pieces
// from all over the batch (k = 8: 706 -> 602 us), and 16 warps keep eight row
// loads per lane in flight (32 warps with four: 628).  A CTA's share is divided
// over its warps in parts, by load (batched_plan.h): cut matrix by matrix from
// warp 0 on, a batch of matrices of fewer slices than warps kept a few warps
// busy (20000 matrices of 32 rows, fp32: k = 1 387 us, 17 in parts; k = 8 524,
// 42).  Large matrices are level cut that way too, and k = 1 takes 4 % less
// time in such segments, whose loops run alike in all warps of a CTA.
// 256 matrices of 1K to 65K rows (0.125G nonzeros, fp32, sigma 256), against
// tiles of slices over all the CTAs that fit: k = 1 468 -> 242, k = 4 1024 ->
// 510, k = 8 2602 -> 582, k = 32 16738 -> 1495 us.
//
// CSR kernel: several waves of the CTAs that fit walk the tiles with a grid
// stride (kCsrWaves);
//   k = 1   tpr lanes per row (tpr in {1,2,4,...,32}, per matrix): lanes
//           stride over the row, shuffle reduction inside the group;
//   k > 1   the tile's columns and values (at most 2048 nonzeros) are staged in
//           shared memory with one coalesced pass; spr groups of G lanes per
//           row read them from there and gather X, shuffle reduction over the
//           groups (same batch: k = 4 918 -> 744, k = 8 1293 -> 916, k = 32 3159 ->
//           1758 us against k lanes of one value each).  Each group keeps two
//           sums and adds four products at a time to one of them in turn (rows
//           of 256 bytes: four sums, of one product each), so that a row's error is no larger than that of eight sums (2 and
//           1000 nonzeros a row, fp32, relative error: 3.6e-7 with two sums
//           that take the products one by one, 1.8e-7 with eight, 8.5e-8 now).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "batched_plan.h"
#include "batched_tune.h"
#include "rvvla_internal.cuh"

namespace rvvla {
namespace {

constexpr int kBThreads = 256;

struct BatchMat {
  const int* Rst;
  const int* Col;
  const void* Val;
  // SELL-C-sigma arrays (mode 1)
  const int* sCl;
  const int* sCs;
  const int* sBs;
  const int* sSBs;
  const uint32_t* sCol;
  const uint32_t* sPerm;
  const void* sVal;
  int64_t x_off, y_off;
  int32_t m, n, mode, tpr;  // tpr: lanes per row (CSR, k = 1)
};

struct BatchTile {
  int32_t mat, first, count, spr;  // spr: lane groups per row, k > 1
};

// SELL: threads of the one CTA per SM (64 or 128 registers each), and the
// pieces of the batch that a CTA takes.
template <class T, int K> constexpr int kSThreads = K == 1 ? 1024 : 512;
constexpr int sell_pieces(int row_bytes) { return row_bytes >= 32 ? 4 : 1; }
// k = 1: segments as long as their busiest warp has at most this much more to
// do than the parts' (256 matrices of 1K to 64K rows, fp32, 1.05: 243 us in
// segments, 251 in parts; 400 of 6000 rows, 1.14: 92 and 79; 800 of 2000, 1.24:
// 67 and 50; 20000 of 32, 26: 387 and 17)
constexpr double kSegSlack = 1.12;

template <class T> struct Vec16;
template <> struct Vec16<float> { using type = float4; };
template <> struct Vec16<double> { using type = double2; };

// N values at p: one 16-byte access (VEC: p is 16-byte aligned), or scalars
template <class T, int N, bool VEC>
__device__ __forceinline__ void load_n(const T* p, T (&v)[N]) {
  if constexpr (VEC && N > 1) {
    using V = typename Vec16<T>::type;
    static_assert(sizeof(V) == N * sizeof(T), "one 16-byte access");
    const V t = *reinterpret_cast<const V*>(p);
    *reinterpret_cast<V*>(v) = t;
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = p[i];
  }
}

template <class T, int N, bool VEC>
__device__ __forceinline__ void store_n(T* p, const T (&v)[N], T alpha, T beta) {
  alignas(16) T o[N];
  if (beta == T(0)) {
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = alpha * v[i];
  } else {
    alignas(16) T y[N];
    load_n<T, N, VEC>(p, y);
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = alpha * v[i] + beta * y[i];
  }
  if constexpr (VEC && N > 1) {
    using V = typename Vec16<T>::type;
    *reinterpret_cast<V*>(p) = *reinterpret_cast<const V*>(o);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = o[i];
  }
}

// X rows are gathered 16 bytes a lane (k > 1).
template <class T, int K>
struct XRows {
  static constexpr int VPL = K == 1 ? 1 : 16 / (int)sizeof(T);  // values per lane
  static constexpr int G = K / VPL;                             // lanes per nonzero
};

// They are re-read across a matrix: kept in L2 against the streams.
__device__ __forceinline__ void gather16(const float* p, float (&v)[4], uint64_t pol) {
  asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p), "l"(pol));
}
__device__ __forceinline__ void gather16(const double* p, double (&v)[2], uint64_t pol) {
  asm("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v[0]), "=d"(v[1]) : "l"(p), "l"(pol));
}
template <class T, int N, bool VEC>
__device__ __forceinline__ void gather_n(const T* p, T (&v)[N], uint64_t pol) {
  if constexpr (VEC && N > 1) {
    gather16(p, v, pol);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = ld_keep(p + i, pol);
  }
}

template <class T>
__device__ __forceinline__ void store_y(T* y, T alpha, T beta, T v) {
  *y = (beta == T(0)) ? alpha * v : alpha * v + beta * *y;
}

// The row pointers of the tile are staged in shared memory first (one
// coalesced load), so no row waits on a dependent row-pointer load.
constexpr int kTileRowsMax = 2048;

template <class T>
__device__ void csr_k1(const BatchMat& A, const BatchTile& t, const int* __restrict__ srst, const T* __restrict__ X,
                       T* __restrict__ Y, T alpha, T beta) {
  const int tpr = A.tpr;
  const int slot = threadIdx.x / tpr, lane = threadIdx.x % tpr, nslots = kBThreads / tpr;
  const T* __restrict__ x = X + A.x_off;
  const T* __restrict__ val = static_cast<const T*>(A.Val);
  const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
  // every group of tpr lanes runs the same number of iterations (row count
  // rounded up), so the sub-warp shuffles below are always convergent
  const int iters = (t.count + nslots - 1) / nslots;
  for (int it = 0; it < iters; ++it) {
    const int rr = it * nslots + slot;
    const bool valid = rr < t.count;
    T s0 = T(0), s1 = T(0);
    if (valid) {
      const int b = srst[rr], e = srst[rr + 1];
      int j = b + lane;
      for (; j + tpr < e; j += 2 * tpr) {
        const int c0 = ld_stream(A.Col + j, pf), c1 = ld_stream(A.Col + j + tpr, pf);
        const T v0 = ld_stream(val + j, pf), v1 = ld_stream(val + j + tpr, pf);
        s0 += v0 * ld_keep(x + c0, pl);
        s1 += v1 * ld_keep(x + c1, pl);
      }
      if (j < e) s0 += ld_stream(val + j, pf) * ld_keep(x + ld_stream(A.Col + j, pf), pl);
    }
    T s = s0 + s1;
    for (int off = tpr >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off, tpr);
    if (valid && lane == 0) store_y(Y + A.y_off + t.first + rr, alpha, beta, s);
  }
}

constexpr int kStageNnz = 2048;  // nonzeros of a k > 1 CSR tile staged in shared memory

template <class T, int K, bool VEC>
__device__ void csr_kn(const BatchMat& A, const BatchTile& t, const int* __restrict__ srst, int* __restrict__ s_col,
                       T* __restrict__ s_val, const T* __restrict__ X, T* __restrict__ Y, T alpha, T beta) {
  using XR = XRows<T, K>;
  constexpr int VPL = XR::VPL, G = XR::G, U = 4;
  const int spr = t.spr, lanes = G * spr, nslots = kBThreads / lanes;
  const int part = threadIdx.x % G, slot = (threadIdx.x / G) % spr, sub = threadIdx.x / lanes;
  const T* __restrict__ x = X + A.x_off + part * VPL;
  const T* __restrict__ val = static_cast<const T*>(A.Val);
  const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
  const int b0 = srst[0], nzt = srst[t.count] - b0;
  // uniform over the CTA (the tile is shared): stage, or read in place (a
  // single row longer than the stage)
  const bool staged = nzt <= kStageNnz;
  if (staged) {
    for (int i = threadIdx.x; i < nzt; i += kBThreads) {
      s_col[i] = ld_stream(A.Col + b0 + i, pf);
      s_val[i] = ld_stream(val + b0 + i, pf);
    }
    __syncthreads();
  }
  // every group runs the same number of iterations, so the shuffles converge
  const int iters = (t.count + nslots - 1) / nslots;
  for (int it = 0; it < iters; ++it) {
    const int rr = it * nslots + sub;
    const bool valid = rr < t.count;
    // the steps' sums go to two accumulators in turn: no chain of roundings is
    // longer than an eighth of the row and a few.  Rows of 256 bytes (at most
    // two groups) take one accumulator per product of a step: as short, and the
    // serial sum of a step is what small batches waited for (100 matrices of 1K
    // to 8K rows, fp64, k = 32: 323 us with it, 282; 400 of 1K to 4K 859 and 772;
    // two sums that take the products one by one, less exact, 265 and 720)
    constexpr int P = G >= 16 ? U : 2;
    T acc[P][VPL];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int i = 0; i < VPL; ++i) acc[p][i] = T(0);
    auto add_step = [&](const T (&t)[VPL]) {
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const T a = acc[0][i] + t[i];
        acc[0][i] = acc[1][i];
        acc[1][i] = a;
      }
    };
    if (valid) {
      const int e = srst[rr + 1] - b0;
      int j = srst[rr] - b0 + slot;
      // rows of 128 bytes and more: whole steps, then one nonzero at a time (a
      // repeated row would cost as much as a new one); narrower ones: idle
      // loads of the last step repeat its first entry
#pragma unroll(G == 8 ? 2 : 1)
      for (; G >= 8 ? j + (U - 1) * spr < e : j < e; j += U * spr) {
        T v[U];
        alignas(16) T xv[U][VPL];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int k = G >= 8 || j + u * spr < e ? j + u * spr : j;
          const int c = staged ? s_col[k] : A.Col[b0 + k];
          v[u] = staged ? s_val[k] : val[b0 + k];
          gather_n<T, VPL, VEC>(x + (int64_t)c * K, xv[u], pl);
        }
        if constexpr (P == U) {
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < VPL; ++i) acc[u][i] += v[u] * xv[u][i];
        } else {
          T t[VPL];
#pragma unroll
          for (int i = 0; i < VPL; ++i) t[i] = v[0] * xv[0][i];
#pragma unroll
          for (int u = 1; u < U; ++u)
            if (G >= 8 || j + u * spr < e) {
#pragma unroll
              for (int i = 0; i < VPL; ++i) t[i] += v[u] * xv[u][i];
            }
          add_step(t);
        }
      }
      T t[VPL];
#pragma unroll
      for (int i = 0; i < VPL; ++i) t[i] = T(0);
      for (; G >= 8 && j < e; j += spr) {
        const int c = staged ? s_col[j] : A.Col[b0 + j];
        const T v = staged ? s_val[j] : val[b0 + j];
        alignas(16) T xv[VPL];
        gather_n<T, VPL, VEC>(x + (int64_t)c * K, xv, pl);
#pragma unroll
        for (int i = 0; i < VPL; ++i) t[i] += v * xv[i];
      }
      if (G >= 8) add_step(t);
    }
    alignas(16) T s[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if constexpr (P == 4) s[i] = (acc[0][i] + acc[1][i]) + (acc[2][i] + acc[3][i]);
      else s[i] = acc[0][i] + acc[1][i];
    }
    for (int off = lanes >> 1; off >= G; off >>= 1)
#pragma unroll
      for (int i = 0; i < VPL; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], off);
    if (valid && slot == 0)
      store_n<T, VPL, VEC>(Y + A.y_off + (int64_t)(t.first + rr) * K + part * VPL, s, alpha, beta);
  }
}

// One SELL slice by one warp.  U columns of values and column indices are
// loaded, then X rows, UX columns of GX rows per lane group at a time.  For k > 1
// four columns' products of a row make a block, and the blocks' sums go to P
// accumulators in turn, which makes the chains of roundings about as short as in
// CSR's sums (error of the batch above, fp32, k = 8: 7.34e-8 with four sums that
// took a product each, 6.84e-8 in blocks; fp64, k = 8, 1061 -> 888 us with
// it).  Rows of 256 bytes leave no registers for that (5830 us against 3815) and
// take one column of all rows at a time into one sum.  For k = 1 the products
// go to four sums.
template <class T, int K, bool VEC>
__device__ __forceinline__ void sell_slice(const BatchMat& A, int sl, const T* __restrict__ x, T* __restrict__ Y,
                                           T alpha, T beta, uint64_t pf, uint64_t pl) {
  using XR = XRows<T, K>;
  constexpr int VPL = XR::VPL, G = XR::G;
  constexpr bool BLOCKS = K > 1 && K * sizeof(T) < 256;
  constexpr int U = G <= 4 ? 8 : 4;
  constexpr int P = K == 1 ? 4 : BLOCKS ? U / 4 : 1;
  constexpr int UX = K == 1 ? U : BLOCKS ? 4 : 1, GX = G == 1 ? 1 : BLOCKS ? 2 : 8;
  constexpr int RS = 32 / G;  // rows per step
  const int lane = threadIdx.x & 31, part = lane % G;
  const T* __restrict__ val = static_cast<const T*>(A.sVal);
  const int* __restrict__ col = reinterpret_cast<const int*>(A.sCol);
  const int h = A.sBs[sl], w = A.sCl[sl];
  const int mine = min(lane, h - 1);  // lanes beyond a short last slice repeat its last row
  const int base = A.sCs[sl] + mine;
  const int row = (int)A.sPerm[A.sSBs[sl] + mine];
  T acc[P][G][VPL];
#pragma unroll
  for (int p = 0; p < P; ++p)
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int i = 0; i < VPL; ++i) acc[p][g][i] = T(0);
  for (int j = 0; j < w; j += U) {
    T v[U];
    int c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {  // columns past the last repeat it and are not added
      const int k = base + min(j + u, w - 1) * h;
      v[u] = ld_stream(val + k, pf);
      c[u] = ld_stream(col + k, pf);
    }
#pragma unroll
    for (int u0 = 0; u0 < U; u0 += UX) {
      if (G > 1 && u0 > 0 && j + u0 >= w) break;  // warp-uniform
#pragma unroll
      for (int g0 = 0; g0 < G; g0 += GX) {
        alignas(16) T xv[UX][GX][VPL];
        T vv[UX][GX];
#pragma unroll
        for (int u = 0; u < UX; ++u)
#pragma unroll
          for (int g = 0; g < GX; ++g) {
            if constexpr (G == 1) {
              vv[u][g] = v[u0 + u];
              gather_n<T, VPL, VEC>(x + (int64_t)c[u0 + u] * K, xv[u][g], pl);
            } else {
              const int src = (g0 + g) * RS + lane / G;
              const int cc = __shfl_sync(0xffffffffu, c[u0 + u], src);
              vv[u][g] = __shfl_sync(0xffffffffu, v[u0 + u], src);
              gather_n<T, VPL, VEC>(x + (int64_t)cc * K + part * VPL, xv[u][g], pl);
            }
          }
#pragma unroll
        for (int g = 0; g < GX; ++g)
#pragma unroll
          for (int i = 0; i < VPL; ++i) {
            if constexpr (BLOCKS) {
              T t = vv[0][g] * xv[0][g][i];
#pragma unroll
              for (int u = 1; u < UX; ++u)
                if (j + u0 + u < w) t += vv[u][g] * xv[u][g][i];
              if (G > 1 || j + u0 < w) acc[u0 / 4][g0 + g][i] += t;
            } else {
#pragma unroll
              for (int u = 0; u < UX; ++u)
                if (j + u0 + u < w) acc[(u0 + u) % P][g0 + g][i] += vv[u][g] * xv[u][g][i];
            }
          }
      }
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    alignas(16) T s[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if constexpr (P == 4) s[i] = (acc[0][g][i] + acc[1][g][i]) + (acc[2][g][i] + acc[3][g][i]);
      else if constexpr (P == 2) s[i] = acc[0][g][i] + acc[1][g][i];
      else s[i] = acc[0][g][i];
    }
    const int rl = g * RS + lane / G;
    const int r = G == 1 ? row : __shfl_sync(0xffffffffu, row, rl);
    if (rl < h) store_n<T, VPL, VEC>(Y + A.y_off + (int64_t)r * K + part * VPL, s, alpha, beta);
  }
}

// The warp's parts.  VEC: X and Y are 16-byte aligned (k > 1; for k = 1 there
// is one form).
template <class T, int K, bool VEC>
__global__ void __launch_bounds__(kSThreads<T, K>, 1)
batched_sell_kernel(const int* __restrict__ share, const BatchPart* __restrict__ parts,
                    const BatchMat* __restrict__ mats, const T* __restrict__ X, T* __restrict__ Y, T alpha, T beta) {
  int warp = threadIdx.x >> 5;
  // a part's indexes are the same in all lanes; told so, the compiler keeps
  // them in uniform registers, which k = 1 and 32 gain by (fp32, the batch
  // above: 278 -> 251 and 1932 -> 1527 us) and k = 4 and 8 lose by (510 and 585
  // -> 507 and 739; fp64 619 and 991 -> 620 and 1015)
  if constexpr (K == 1 || K == 32) warp = __shfl_sync(0xffffffffu, warp, 0);
  const int at = blockIdx.x * (kSThreads<T, K> / 32) + warp;
  const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
  const int p1 = share[at + 1];
  for (int pi = share[at]; pi < p1; ++pi) {
    const BatchPart p = parts[pi];
    const BatchMat A = mats[p.mat];
    const T* x = X + A.x_off;
    for (int u = p.first; u < p.end; ++u) sell_slice<T, K, VEC>(A, u, x, Y, alpha, beta, pf, pl);
  }
}

// The CTA's segments, k = 1.
template <class T>
__global__ void __launch_bounds__(kSThreads<T, 1>, 1)
batched_seg_kernel(const int* __restrict__ share, const BatchSeg* __restrict__ segs,
                   const BatchMat* __restrict__ mats, const T* __restrict__ X, T* __restrict__ Y, T alpha, T beta) {
  static_assert(kSThreads<T, 1> == 32 * kSegWarps, "a segment is cut for the CTA's warps");
  const int warp = threadIdx.x >> 5;
  const uint64_t pf = policy_evict_first(), pl = policy_evict_last();
  const int s1 = share[blockIdx.x + 1];
  for (int si = share[blockIdx.x]; si < s1; ++si) {  // no step of a segment spans warps
    const BatchSeg& sg = segs[si];
    const BatchMat& A = mats[sg.mat];
    const int u1 = sg.first[warp + 1];
    const T* x = X + A.x_off;
    for (int u = sg.first[warp]; u < u1; ++u) sell_slice<T, 1, true>(A, u, x, Y, alpha, beta, pf, pl);
  }
}

// Five CTAs per SM in fp64 (k = 4: 1232 us for the batch above with the four
// that the registers allow otherwise, 1120 with five and a little spilled).
template <class T, int K, bool VEC>
__global__ void __launch_bounds__(kBThreads, K > 1 && sizeof(T) == 8 ? 5 : 0)
batched_kernel(int64_t ntiles, const BatchTile* __restrict__ tiles, const BatchMat* __restrict__ mats,
               const T* __restrict__ X, T* __restrict__ Y, T alpha, T beta) {
  // per tile: the matrix entry and the tile's row pointers are copied to
  // shared memory once, then used by all warps
  __shared__ int srst[kTileRowsMax + 1];
  __shared__ int s_col[K > 1 ? kStageNnz : 1];
  __shared__ T s_val[K > 1 ? kStageNnz : 1];
  __shared__ __align__(16) unsigned char sAraw[sizeof(BatchMat)];
  const BatchMat& A = *reinterpret_cast<const BatchMat*>(sAraw);
  static_assert(sizeof(BatchMat) % 8 == 0, "BatchMat is copied as 8-byte words");
  for (int64_t ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
    const BatchTile t = tiles[ti];
    __syncthreads();  // the previous tile is done with the shared copies
    if (threadIdx.x < (int)(sizeof(BatchMat) / 8))
      reinterpret_cast<uint64_t*>(sAraw)[threadIdx.x] =
          reinterpret_cast<const uint64_t*>(mats + t.mat)[threadIdx.x];
    __syncthreads();
    for (int i = threadIdx.x; i <= t.count; i += kBThreads) srst[i] = A.Rst[t.first + i];
    __syncthreads();
    if constexpr (K == 1) csr_k1<T>(A, t, srst, X, Y, alpha, beta);
    else csr_kn<T, K, VEC>(A, t, srst, s_col, s_val, X, Y, alpha, beta);
  }
}

constexpr int64_t kTileWork = 8192;  // k = 1 CSR tile: nonzeros + rows

// CSR CTAs per resident one, at most; a CTA per tile for X rows of 128 bytes and
// more.  CTAs that walk a long list with a grid stride drift apart and spread over
// more matrices than L2 holds the X of; new CTAs take the tiles in order.  1024
// matrices of 1K to 64K rows, k = 32, fp32: 11.7 ms with the resident CTAs, 10.6,
// 8.3 and 7.6 with 4 and 16 times as many and one per tile; 256 of them, fp64, 4.0,
// 3.8, 3.0, 2.8 ms.  Narrower rows gain less and lose a little to a CTA per tile
// (256, fp32: k = 1 533, 516, 489, 484 us, k = 4 751, 756, 742, 759, k = 8 923,
// 947, 915, 934).
constexpr int64_t kCsrWaves = 16;

int default_tpr(double avg) {
  int t = 1;
  while (t < 32 && t < avg) t <<= 1;
  return std::max(1, t / 2);
}

// Lanes per nonzero.
int lanes_nz(int k, int vb) { return k == 1 ? 1 : k * vb / 16; }

// Lane groups per CSR row for k > 1: at least eight nonzeros per group (fewer
// leave more of the four loads per lane and step idle: k = 4 / 8 fp32, the
// batch above: 907 / 1168 us with two per group, 759 / 1010 with eight), but in
// a tile with a long row enough for at most 32 nonzeros per group, which bounds
// both the time that row takes and the roundings in its sums.
int default_spr(double avg, int64_t longest, int lanes) {
  int t = 1;
  while (2 * t * lanes <= 32 && (16 * t <= avg || 32 * t < longest)) t <<= 1;
  return t;
}

template <class T, int K, bool VEC>
int launch_k(const rvvla_batch* B, T alpha, const T* X, T beta, T* Y, cudaStream_t st) {
  const auto* mats = static_cast<const BatchMat*>(B->mats);
  const auto* tiles = static_cast<const BatchTile*>(B->tiles);
  const int64_t ncsr = B->ntiles - B->sell_segs - B->sell_parts;
  if (ncsr > 0) {
    batched_kernel<T, K, VEC><<<B->grid, kBThreads, 0, st>>>(ncsr, tiles, mats, X, Y, alpha, beta);
    RVVLA_LAUNCHED("batched_kernel");
  }
  // after the tiles: the SELL work, then its shares
  const auto* parts = reinterpret_cast<const BatchPart*>(tiles + ncsr);
  const auto* segs = reinterpret_cast<const BatchSeg*>(parts + B->sell_parts);
  const auto* share = reinterpret_cast<const int*>(segs + B->sell_segs);
  if (B->sell_parts > 0) {
    batched_sell_kernel<T, K, VEC><<<sm_count(), kSThreads<T, K>, 0, st>>>(share, parts, mats, X, Y, alpha, beta);
    RVVLA_LAUNCHED("batched_sell_kernel");
  }
  if constexpr (K == 1) {
    if (B->sell_segs > 0) {
      batched_seg_kernel<T><<<sm_count(), kSThreads<T, 1>, 0, st>>>(share, segs, mats, X, Y, alpha, beta);
      RVVLA_LAUNCHED("batched_seg_kernel");
    }
  }
  return RVVLA_OK;
}

template <class T, int K>
int launch_v(const rvvla_batch* B, T alpha, const T* X, T beta, T* Y, cudaStream_t st) {
  if constexpr (K > 1) {
    if ((uintptr_t)X % 16 != 0 || (uintptr_t)Y % 16 != 0) return launch_k<T, K, false>(B, alpha, X, beta, Y, st);
  }
  return launch_k<T, K, true>(B, alpha, X, beta, Y, st);
}

template <class T>
int batched_launch(const rvvla_batch* B, T alpha, const T* X, T beta, T* Y, cudaStream_t st) {
  if (!B) return fail(RVVLA_ERR_INVALID_ARG, "batched_spmv: null plan");
  if (B->val_bytes != (int)sizeof(T)) return fail(RVVLA_ERR_INVALID_ARG, "batched_spmv: value type differs from the plan");
  if (B->ntiles == 0) return RVVLA_OK;
  if ((B->x_len > 0 && !X) || (B->y_len > 0 && !Y)) return fail(RVVLA_ERR_INVALID_ARG, "batched_spmv: null vectors");
  switch (B->k) {
    case 1: return launch_v<T, 1>(B, alpha, X, beta, Y, st);
    case 4: return launch_v<T, 4>(B, alpha, X, beta, Y, st);
    case 8: return launch_v<T, 8>(B, alpha, X, beta, Y, st);
    case 32: return launch_v<T, 32>(B, alpha, X, beta, Y, st);
    default: return fail(RVVLA_ERR_INVALID_ARG, "batched_spmv: bad k in plan");
  }
}

template <class T>
int resident_ctas(int k) {
  int per_sm = 1;
  auto kern = k == 1   ? batched_kernel<T, 1, true>
              : k == 4 ? batched_kernel<T, 4, true>
              : k == 8 ? batched_kernel<T, 8, true>
                       : batched_kernel<T, 32, true>;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBThreads, 0) != cudaSuccess) per_sm = 1;
  return std::max(per_sm, 1);
}

// Times one plan: one warm-up launch, then the best of three (CUDA events on
// `st`, zeroed X from the stream-ordered pool).
int time_plan(const rvvla_batch& B, cudaStream_t st, double* ms) {
  *ms = 0.0;
  if (B.ntiles == 0) return RVVLA_OK;
  const size_t vb = (size_t)B.val_bytes;
  Scratch sx, sy;
  RVVLA_CUDA(sx.alloc(std::max<int64_t>(B.x_len, 1) * vb, st));
  RVVLA_CUDA(sy.alloc(std::max<int64_t>(B.y_len, 1) * vb, st));
  RVVLA_CUDA(cudaMemsetAsync(sx.p, 0, std::max<int64_t>(B.x_len, 1) * vb, st));
  cudaEvent_t e0, e1;
  RVVLA_CUDA(cudaEventCreate(&e0));
  RVVLA_CUDA(cudaEventCreate(&e1));
  double best = 1e30;
  int rc = RVVLA_OK;
  for (int it = 0; it < 4 && rc == RVVLA_OK; ++it) {
    cudaEventRecord(e0, st);
    rc = (vb == 8) ? batched_launch<double>(&B, 1.0, sx.as<double>(), 0.0, sy.as<double>(), st)
                   : batched_launch<float>(&B, 1.f, sx.as<float>(), 0.f, sy.as<float>(), st);
    cudaEventRecord(e1, st);
    if (cudaEventSynchronize(e1) != cudaSuccess) rc = fail(RVVLA_ERR_CUDA, "autotune: launch failed");
    float t = 0.f;
    cudaEventElapsedTime(&t, e0, e1);
    if (it > 0) best = std::min(best, (double)t);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *ms = best;
  return rc;
}

struct BatchGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int kernels = 0;
};

}  // namespace
}  // namespace rvvla

using namespace rvvla;

extern "C" {

void rvvla_batched_free(rvvla_batch_owned* b) {
  if (!b) return;
  if (b->sell)
    for (int64_t i = 0; i < b->nmats; ++i) rvvla_sell_free(&b->sell[i]);
  if (b->mats) cudaFree(b->mats);
  if (b->tiles) cudaFree(b->tiles);
  std::free(b->x_off);
  std::free(b->y_off);
  std::free(b->sell);
  std::memset(b, 0, sizeof(*b));
}

int rvvla_batched_plan(const rvvla_crs* mats, int64_t count, int val_bytes, int k, const int32_t* mode,
                       const int32_t* param, rvvla_batch_owned* out, void* stream) {
  if (!out) return fail(RVVLA_ERR_INVALID_ARG, "batched_plan: null output");
  std::memset(out, 0, sizeof(*out));
  if (count < 0 || (count > 0 && !mats)) return fail(RVVLA_ERR_INVALID_ARG, "batched_plan: bad matrix list");
  if (val_bytes != 4 && val_bytes != 8) return fail(RVVLA_ERR_INVALID_ARG, "batched_plan: val_bytes must be 4 or 8");
  if (k != 1 && k != 4 && k != 8 && k != 32) return fail(RVVLA_ERR_INVALID_ARG, "batched_plan: k must be 1, 4, 8 or 32");
  cudaStream_t st = as_stream(stream);
  int rc = RVVLA_OK;
  std::vector<BatchMat> tab((size_t)count);
  std::vector<BatchTile> tiles;
  std::vector<SliceUnit> slices;
  out->x_off = static_cast<int64_t*>(std::calloc((size_t)count + 1, sizeof(int64_t)));
  out->y_off = static_cast<int64_t*>(std::calloc((size_t)count + 1, sizeof(int64_t)));
  out->sell = static_cast<rvvla_sell_owned*>(std::calloc((size_t)std::max<int64_t>(count, 1), sizeof(rvvla_sell_owned)));
  out->nmats = count;
  if (!out->x_off || !out->y_off || !out->sell) {
    rvvla_batched_free(out);
    return fail(RVVLA_ERR_CUDA, "batched_plan: host allocation failed");
  }
  std::vector<int> Rst;
  for (int64_t i = 0; i < count && rc == RVVLA_OK; ++i) {
    const rvvla_crs& A = mats[i];
    if (A.m < 0 || A.n < 0 || A.nz < 0 || A.m >= INT32_MAX || A.n >= INT32_MAX || A.nz >= INT32_MAX ||
        (A.m > 0 && !A.Rst) || (A.nz > 0 && (!A.Col || !A.Val))) {
      rc = fail(RVVLA_ERR_INVALID_ARG, "batched_plan: matrix " + std::to_string(i) + " has bad sizes or arrays");
      break;
    }
    BatchMat& b = tab[(size_t)i];
    std::memset(&b, 0, sizeof(b));
    b.Rst = A.Rst; b.Col = A.Col; b.Val = A.Val;
    b.m = (int32_t)A.m; b.n = (int32_t)A.n;
    b.x_off = out->x_off[i];
    b.y_off = out->y_off[i];
    out->x_off[i + 1] = out->x_off[i] + A.n * k;
    out->y_off[i + 1] = out->y_off[i] + A.m * k;
    if (A.m == 0) continue;
    const int md = mode ? mode[i] : 0;
    const double avg = (double)A.nz / (double)A.m;
    if (md == 0) {
      b.mode = 0;
      Rst.resize((size_t)A.m + 1);  // the tiles are cut on the host
      if (cudaMemcpyAsync(Rst.data(), A.Rst, (A.m + 1) * sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess) {
        rc = fail(RVVLA_ERR_CUDA, "batched_plan: reading row pointers failed");
        break;
      }
      const int tpr = (param && param[i] > 0) ? param[i] : default_tpr(avg);
      if (tpr > 32 || (tpr & (tpr - 1))) {
        rc = fail(RVVLA_ERR_INVALID_ARG, "batched_plan: threads per row must be a power of two <= 32");
        break;
      }
      b.tpr = tpr;
      const int lanes = lanes_nz(k, val_bytes), lanes_row = (k == 1) ? tpr : default_spr(avg, 0, lanes) * lanes;
      // tiles of whole rows: k = 1 at most kTileWork nonzeros and 8 row
      // passes of the CTA; k > 1 at most the staged nonzeros and 32 passes
      const int64_t max_rows = std::min<int64_t>((int64_t)(kBThreads / lanes_row) * (k == 1 ? 8 : 32), kTileRowsMax);
      const int64_t max_work = k == 1 ? kTileWork : kStageNnz;
      int64_t r0 = 0;
      while (r0 < A.m) {
        int64_t r1 = r0, work = 0, longest = 0;
        while (r1 < A.m && r1 - r0 < max_rows) {
          const int64_t wr = (int64_t)Rst[(size_t)r1 + 1] - Rst[(size_t)r1] + (k == 1 ? 1 : 0);
          if (r1 > r0 && work + wr > max_work) break;
          work += wr;
          longest = std::max(longest, wr);
          ++r1;
        }
        tiles.push_back({(int32_t)i, (int32_t)r0, (int32_t)(r1 - r0), k == 1 ? tpr : default_spr(avg, longest, lanes)});
        r0 = r1;
      }
    } else if (md == 1) {
      b.mode = 1;
      const int sigma = (param && param[i] > 0) ? param[i] : 256;
      rvvla_crs src = A;
      src.plan = nullptr;
      src.plan_tiles = 0;
      src.plan_kind = 0;
      rc = rvvla_sell_build(&src, val_bytes, 32, sigma, &out->sell[i], stream);
      if (rc) break;
      const rvvla_sell& s = out->sell[i].h;
      b.sCl = s.vCl; b.sCs = s.vCs; b.sBs = s.vBs; b.sSBs = s.vSBs;
      b.sCol = s.vCol; b.sPerm = s.vPerm; b.sVal = s.vVal;
      std::vector<int> Cl((size_t)s.cnt_b);
      if (s.cnt_b && (cudaMemcpy(Cl.data(), s.vCl, s.cnt_b * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)) {
        rc = fail(RVVLA_ERR_CUDA, "batched_plan: reading slice widths failed");
        break;
      }
      for (int64_t q = 0; q < s.cnt_b; ++q) slices.push_back({(int32_t)i, (int32_t)q, (int64_t)Cl[(size_t)q] + 2});
    } else {
      rc = fail(RVVLA_ERR_INVALID_ARG, "batched_plan: mode must be 0 (CSR) or 1 (SELL)");
      break;
    }
  }
  if (rc) {
    std::string keep = rvvla_last_error();
    rvvla_batched_free(out);
    set_error(keep);
    return rc;
  }
  rvvla_batch& h = out->h;
  h.count = count;
  h.k = k;
  h.val_bytes = val_bytes;
  h.x_len = out->x_off[count];
  h.y_len = out->y_off[count];
  const int warps = (k == 1 ? kSThreads<float, 1> : kSThreads<float, 8>) / 32, pieces = sell_pieces(k * val_bytes);
  SlicePlan sp = plan_parts(slices, sm_count(), pieces, warps);
  if (k == 1) {
    SlicePlan sg = plan_segments(slices, sm_count(), pieces);
    if ((double)sg.busiest <= kSegSlack * (double)sp.busiest) sp = std::move(sg);
  }
  h.sell_segs = (int32_t)sp.segs.size();
  h.sell_parts = (int32_t)sp.parts.size();
  h.ntiles = (int64_t)tiles.size() + h.sell_segs + h.sell_parts;
  auto fail_cuda = [&](cudaError_t e, const char* where) {
    const int r = cuda_fail(e, where);
    std::string keep = rvvla_last_error();
    rvvla_batched_free(out);
    set_error(keep);
    return r;
  };
  cudaError_t e;
  if ((e = cudaMalloc(&out->mats, std::max<size_t>(tab.size(), 1) * sizeof(BatchMat))) != cudaSuccess)
    return fail_cuda(e, "cudaMalloc(mats)");
  // the CSR tiles, the SELL parts, the SELL segments, their shares
  const std::pair<const void*, size_t> lists[] = {{tiles.data(), tiles.size() * sizeof(BatchTile)},
                                                  {sp.parts.data(), sp.parts.size() * sizeof(BatchPart)},
                                                  {sp.segs.data(), sp.segs.size() * sizeof(BatchSeg)},
                                                  {sp.share.data(), sp.share.size() * sizeof(int32_t)}};
  size_t bytes = 0;
  for (const auto& l : lists) bytes += l.second;
  if ((e = cudaMalloc(&out->tiles, bytes)) != cudaSuccess) return fail_cuda(e, "cudaMalloc(tiles)");
  if (!tab.empty() &&
      (e = cudaMemcpyAsync(out->mats, tab.data(), tab.size() * sizeof(BatchMat), cudaMemcpyHostToDevice, st)) != cudaSuccess)
    return fail_cuda(e, "cudaMemcpyAsync(mats)");
  char* to = static_cast<char*>(out->tiles);
  for (const auto& l : lists) {
    if (l.second && (e = cudaMemcpyAsync(to, l.first, l.second, cudaMemcpyHostToDevice, st)) != cudaSuccess)
      return fail_cuda(e, "cudaMemcpyAsync(tiles)");
    to += l.second;
  }
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return fail_cuda(e, "cudaStreamSynchronize");
  // grid of the CSR kernel: every SM filled with as many CTAs as fit, some times over
  const int per_sm = (val_bytes == 8) ? resident_ctas<double>(k) : resident_ctas<float>(k);
  // (kCsrWaves)
  const int64_t most = k * val_bytes >= 128 ? INT32_MAX : (int64_t)sm_count() * per_sm * kCsrWaves;
  h.grid = (int32_t)std::max<int64_t>(1, std::min<int64_t>(most, (int64_t)tiles.size()));
  h.block = kBThreads;
  h.mats = out->mats;
  h.tiles = out->tiles;
  return RVVLA_OK;
}

int rvvla_batched_spmv_f64(const rvvla_batch* B, double alpha, const double* X, double beta, double* Y, void* stream) {
  return batched_launch<double>(B, alpha, X, beta, Y, as_stream(stream));
}

int rvvla_batched_spmv_f32(const rvvla_batch* B, float alpha, const float* X, float beta, float* Y, void* stream) {
  return batched_launch<float>(B, alpha, X, beta, Y, as_stream(stream));
}

int rvvla_batched_graph(const rvvla_batch* B, double alpha, const void* X, double beta, void* Y, void* stream,
                        void** graph) {
  if (!B || !graph) return fail(RVVLA_ERR_INVALID_ARG, "batched_graph: null argument");
  *graph = nullptr;
  cudaStream_t st = as_stream(stream);
  if (!st) return fail(RVVLA_ERR_INVALID_ARG, "batched_graph: capture needs a non-default stream");
  auto* g = new BatchGraph();
  g->kernels = (B->ntiles > B->sell_segs + B->sell_parts ? 1 : 0) + (B->sell_segs + B->sell_parts > 0 ? 1 : 0);
  const cudaError_t eb = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
  if (eb != cudaSuccess) {
    delete g;
    return cuda_fail(eb, "cudaStreamBeginCapture");
  }
  const int rc = (B->val_bytes == 8)
                     ? batched_launch<double>(B, alpha, static_cast<const double*>(X), beta, static_cast<double*>(Y), st)
                     : batched_launch<float>(B, (float)alpha, static_cast<const float*>(X), (float)beta,
                                             static_cast<float*>(Y), st);
  const cudaError_t ec = cudaStreamEndCapture(st, &g->graph);
  if (rc || ec != cudaSuccess) {
    if (g->graph) cudaGraphDestroy(g->graph);
    delete g;
    return rc ? rc : cuda_fail(ec, "cudaStreamEndCapture");
  }
  const cudaError_t ei = cudaGraphInstantiate(&g->exec, g->graph, 0);
  if (ei != cudaSuccess) {
    cudaGraphDestroy(g->graph);
    delete g;
    return cuda_fail(ei, "cudaGraphInstantiate");
  }
  *graph = g;
  return RVVLA_OK;
}

int rvvla_batched_graph_launch(void* graph, void* stream) {
  if (!graph) return fail(RVVLA_ERR_INVALID_ARG, "batched_graph_launch: null graph");
  auto* g = static_cast<BatchGraph*>(graph);
  RVVLA_CUDA(cudaGraphLaunch(g->exec, as_stream(stream)));
  count_launch((uint64_t)g->kernels);
  return RVVLA_OK;
}

void rvvla_batched_graph_free(void* graph) {
  if (!graph) return;
  auto* g = static_cast<BatchGraph*>(graph);
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  delete g;
}

int rvvla_batched_autotune(const rvvla_crs* mats, int64_t count, int val_bytes, int k, int32_t* mode, int32_t* param,
                           double* tuned_ms, void* stream) {
  if (count < 0 || (count > 0 && (!mats || !mode || !param)))
    return fail(RVVLA_ERR_INVALID_ARG, "batched_autotune: null argument");
  if (tuned_ms) *tuned_ms = 0.0;
  cudaStream_t st = as_stream(stream);
  // groups by average row length: [0,2), [2,4), [4,8), ... [128, inf)
  constexpr int kGroups = 8;
  std::vector<std::vector<int64_t>> groups(kGroups);
  for (int64_t i = 0; i < count; ++i) {
    const double avg = mats[i].m > 0 ? (double)mats[i].nz / (double)mats[i].m : 0.0;
    int g = 0;
    while (g + 1 < kGroups && avg >= (double)(2 << g)) ++g;
    groups[(size_t)g].push_back(i);
  }
  std::vector<TuneCand> cands;
  if (k == 1)
    for (int t = 1; t <= 32; t <<= 1) cands.push_back({0, t});
  else
    cands.push_back({0, 0});
  cands.push_back({1, 32});
  cands.push_back({1, 256});
  std::vector<TuneCand> pick;
  double total = 0.0;
  const int rc = tune_layouts(
      groups, count, cands,
      [&](const std::vector<int64_t>& ids, const std::vector<TuneCand>& of, double* ms) {
        std::vector<rvvla_crs> sub;
        std::vector<int32_t> md, pr;
        for (size_t i = 0; i < ids.size(); ++i) {
          sub.push_back(mats[ids[i]]);
          md.push_back(of[i].mode);
          pr.push_back(of[i].param);
        }
        rvvla_batch_owned plan;
        int r = rvvla_batched_plan(sub.data(), (int64_t)sub.size(), val_bytes, k, md.data(), pr.data(), &plan, stream);
        if (r) return r;
        r = time_plan(plan.h, st, ms);
        rvvla_batched_free(&plan);
        return r;
      },
      pick, &total);
  if (rc) return rc;
  for (int64_t i = 0; i < count; ++i) {
    mode[i] = pick[(size_t)i].mode;
    param[i] = pick[(size_t)i].param;
  }
  if (tuned_ms) *tuned_ms = total;
  return RVVLA_OK;
}

}  // extern "C"
