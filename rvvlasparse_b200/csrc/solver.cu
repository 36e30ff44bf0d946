// solver.cu — conjugate gradients (symmetric positive definite A) and
// BiCGStab (general square A) over the CRS kernels (no reference
// counterpart: callers of the SpMV path).
//
// A CG iteration is four launches on the caller's stream and no host
// synchronisation:
//   1. q = A p with the fused dot: the CRS lane-run kernel adds p[row] * v
//      for every row piece v it stores or carries into a per-warp partial,
//      so p^T A p needs no second pass over q;
//   2. the rows that cross warps, and the sum of those partials: p.q;
//   3. r -= alpha q with alpha = r.r / p.q, and the new r.r in the same pass;
//   4. x += alpha p and p = r + beta p, beta = r.r(new) / r.r(old), one read of
//      p for both.
// (2) and (3) add their blocks' partials in the block that finishes last.
// Bound by HBM: the product (see crs_run.cuh) and 8 vectors a pass.  5-point
// Laplacian 2048^2, fp64: 167 us per iteration with the scalars in kernels of
// their own and x updated beside r (9 vectors), 155 with four launches, 147
// with each launch chained to the one before (grid_chain: it starts while that
// one drains), 138 with the product in CTAs of four warps.
// The scalars live in device memory; every check_every iterations the host
// reads r.r once to test ||r|| <= rtol ||b||.  All reductions run in a fixed
// order, so a solve is bitwise reproducible.
#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>

#include "rvvla_internal.cuh"

namespace rvvla {

int crs_spmv_dot_f64(const rvvla_crs* A, const double* p, double* q, const CrsDot& dot, cudaStream_t st);
int crs_spmv_dot_f32(const rvvla_crs* A, const float* p, float* q, const CrsDot& dot, cudaStream_t st);
int64_t crs_warp_count(int64_t nz);

namespace {

struct CgScalars {
  double rr[2];  // r.r of the residuals of even and odd iterations
  double pq;     // p.(A p)
  double bb;     // b.b
  unsigned ticket_dot, ticket_rr;  // blocks done, of the kernels that add partials (0 between launches)
};

constexpr int kRedThreads = 1024;
constexpr int kUpdThreads = 256;

// Sum of v[0..n) by one block: thread t adds t, t + 1024, ... in order, then
// a fixed tree in shared memory.
template <class T>
__device__ double block_sum(const T* __restrict__ v, int64_t n) {
  __shared__ double sh[kRedThreads];
  double a = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += kRedThreads) a += (double)v[i];
  sh[threadIdx.x] = a;
  __syncthreads();
  for (int d = kRedThreads / 2; d > 0; d >>= 1) {
    if ((int)threadIdx.x < d) sh[threadIdx.x] += sh[threadIdx.x + d];
    __syncthreads();
  }
  return sh[0];
}

// per-block partial of u.v over a grid-stride loop (fixed grid: fixed order)
__device__ void block_partial(double a, double* __restrict__ part) {
  __shared__ double sh[kUpdThreads];
  sh[threadIdx.x] = a;
  __syncthreads();
  for (int d = kUpdThreads / 2; d > 0; d >>= 1) {
    if ((int)threadIdx.x < d) sh[threadIdx.x] += sh[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

template <class T>
__global__ void __launch_bounds__(kUpdThreads) cg_dot_kernel(int64_t n, const T* __restrict__ u,
                                                             const T* __restrict__ v, double* __restrict__ part) {
  double a = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kUpdThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kUpdThreads)
    a += (double)u[i] * (double)v[i];
  block_partial(a, part);
}

__global__ void __launch_bounds__(kRedThreads) cg_set_kernel(const double* __restrict__ part, int64_t n,
                                                             CgScalars* s, int which) {
  const double v = block_sum(part, n);
  if (threadIdx.x == 0) {
    if (which == 0) {
      s->rr[0] = v;
      s->ticket_dot = s->ticket_rr = 0u;
    } else {
      s->bb = v;
    }
  }
}

__device__ __forceinline__ double cg_alpha(const CgScalars* s, int cur) {
  return s->pq != 0.0 ? s->rr[cur] / s->pq : 0.0;
}

// r -= alpha q and the new r.r: the block that finishes last adds the blocks'
// partials in a fixed order.
template <class T>
__global__ void __launch_bounds__(kUpdThreads) cg_update_kernel(int64_t n, T* r, const T* q, CgScalars* s, int cur,
                                                                double* part) {
  __shared__ bool last;
  grid_chain();
  // r and q start 16-byte aligned: 16 bytes a thread, two loads of each in flight
  constexpr int E = 16 / (int)sizeof(T);
  struct alignas(16) Vec {
    T v[E];
  };
  const T alpha = (T)cg_alpha(s, cur);
  double a = 0.0;
  const int64_t nv = n / E, step = (int64_t)gridDim.x * kUpdThreads;
  Vec* rv = reinterpret_cast<Vec*>(r);
  const Vec* qv = reinterpret_cast<const Vec*>(q);
  auto upd = [&](Vec& ri, const Vec& qi) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      ri.v[e] -= alpha * qi.v[e];
      a += (double)ri.v[e] * (double)ri.v[e];
    }
  };
  int64_t i = (int64_t)blockIdx.x * kUpdThreads + threadIdx.x;
  for (; i + step < nv; i += 2 * step) {
    Vec r0 = rv[i], r1 = rv[i + step];
    const Vec q0 = qv[i], q1 = qv[i + step];
    upd(r0, q0);
    upd(r1, q1);
    rv[i] = r0;
    rv[i + step] = r1;
  }
  if (i < nv) {
    Vec r0 = rv[i];
    upd(r0, qv[i]);
    rv[i] = r0;
  }
  if (blockIdx.x == 0 && threadIdx.x < n - nv * E) {  // the last n mod E
    const int64_t k = nv * E + threadIdx.x;
    const T rk = r[k] - alpha * q[k];
    r[k] = rk;
    a += (double)rk * (double)rk;
  }
  block_partial(a, part);
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&s->ticket_rr, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kUpdThreads) t += __ldcg(part + i);
  __shared__ double sh[kUpdThreads];
  sh[threadIdx.x] = t;
  __syncthreads();
  for (int d = kUpdThreads / 2; d > 0; d >>= 1) {
    if ((int)threadIdx.x < d) sh[threadIdx.x] += sh[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    s->rr[cur ^ 1] = sh[0];
    s->ticket_rr = 0u;
  }
}

template <class T>
__global__ void __launch_bounds__(kRedThreads) sum_to_kernel(const T* __restrict__ part, int64_t n, T* out) {
  const double v = block_sum(part, n);
  if (threadIdx.x == 0) *out = (T)v;
}

template <class T>
__global__ void store_dot_kernel(const double* __restrict__ v, T* __restrict__ out) { *out = (T)*v; }

int64_t dot_blocks(int64_t nw) { return (2 * nw + 255) / 256; }  // crs_dot_fixup_kernel's

template <class T>
int spmv_dot_impl(const rvvla_crs* A, const T* x, T* y, T* dot, cudaStream_t st) {
  if (!A || !x || !y || !dot) return fail(RVVLA_ERR_INVALID_ARG, "crs_spmv_dot: null argument");
  if (A->m != A->n) return fail(RVVLA_ERR_INVALID_ARG, "crs_spmv_dot: A must be square");
  if (A->m == 0 || A->nz == 0) {  // y = 0, dot = 0
    if (A->m > 0) RVVLA_CUDA(cudaMemsetAsync(y, 0, (size_t)A->m * sizeof(T), st));
    RVVLA_CUDA(cudaMemsetAsync(dot, 0, sizeof(T), st));
    return RVVLA_OK;
  }
  const int64_t nw = crs_warp_count(A->nz);
  const size_t partb = ((size_t)nw * sizeof(T) + 255) / 256 * 256;
  const size_t sumb = (size_t)dot_blocks(nw) * sizeof(double);
  Scratch sc;
  RVVLA_CUDA(sc.alloc_kept(partb + sumb + 256, st));
  char* base = sc.as<char>();
  double* out = reinterpret_cast<double*>(base + partb + sumb);
  CrsDot cd{base, reinterpret_cast<double*>(base + partb), reinterpret_cast<unsigned*>(out + 1), out};
  RVVLA_CUDA(cudaMemsetAsync(cd.ticket, 0, sizeof(unsigned), st));
  const int rc = std::is_same<T, double>::value
                     ? crs_spmv_dot_f64(A, reinterpret_cast<const double*>(x), reinterpret_cast<double*>(y), cd, st)
                     : crs_spmv_dot_f32(A, reinterpret_cast<const float*>(x), reinterpret_cast<float*>(y), cd, st);
  if (rc) return rc;
  store_dot_kernel<T><<<1, 1, 0, st>>>(out, dot);
  RVVLA_LAUNCHED("store_dot_kernel");
  return RVVLA_OK;
}

// x += alpha p, p = r + beta p: the x update shares the read of p.
template <class T>
__global__ void cg_xp_kernel(int64_t n, T* x, T* p, const T* r, const CgScalars* s, int cur) {
  grid_chain();
  const T alpha = (T)cg_alpha(s, cur);
  const T beta = (T)(s->rr[cur] != 0.0 ? s->rr[cur ^ 1] / s->rr[cur] : 0.0);
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const T pi = p[i], ri = r[i], xi = x[i];  // all loads before the stores
    x[i] = xi + alpha * pi;
    p[i] = ri + beta * pi;
  }
}

template <class T>
int cg_impl(const rvvla_crs* A, const T* b, T* x, int64_t max_iter, double rtol, int64_t check_every, int64_t* iters,
            double* rel_res, cudaStream_t st) {
  if (!A || !b || !x || !iters || !rel_res) return fail(RVVLA_ERR_INVALID_ARG, "cg: null argument");
  if (A->m != A->n || A->m <= 0) return fail(RVVLA_ERR_INVALID_ARG, "cg: A must be square and non-empty");
  if (max_iter < 0 || check_every <= 0 || !(rtol >= 0.0))
    return fail(RVVLA_ERR_INVALID_ARG, "cg: bad iteration limits");
  if (A->nz == 0 || !A->plan || (A->plan_kind != 1 && A->plan_kind != 2))
    return fail(RVVLA_ERR_INVALID_ARG, "cg: A needs nonzeros and an analysed plan (rvvla_crs_analyze)");
  const int64_t n = A->n;
  const int64_t nw = crs_warp_count(A->nz);
  const int upd_blocks = (int)std::min<int64_t>((n + kUpdThreads - 1) / kUpdThreads, (int64_t)sm_count() * 8);
  Scratch sc;
  const size_t vec = ((size_t)n * sizeof(T) + 255) / 256 * 256;
  const size_t partb = ((size_t)std::max<int64_t>(nw, 1) * sizeof(T) + 255) / 256 * 256;
  const size_t sumb = ((size_t)dot_blocks(nw) * sizeof(double) + 255) / 256 * 256;
  const size_t rrb = ((size_t)upd_blocks * sizeof(double) + 255) / 256 * 256;
  RVVLA_CUDA(sc.alloc_kept(3 * vec + partb + sumb + rrb + sizeof(CgScalars), st));
  char* base = sc.as<char>();
  T* r = reinterpret_cast<T*>(base);
  T* p = reinterpret_cast<T*>(base + vec);
  T* q = reinterpret_cast<T*>(base + 2 * vec);
  double* rrp = reinterpret_cast<double*>(base + 3 * vec + partb + sumb);
  CgScalars* s = reinterpret_cast<CgScalars*>(base + 3 * vec + partb + sumb + rrb);
  const CrsDot cd{base + 3 * vec, reinterpret_cast<double*>(base + 3 * vec + partb), &s->ticket_dot, &s->pq};
  // r = b - A x, p = r, r.r, b.b
  RVVLA_CUDA(cudaMemcpyAsync(r, b, (size_t)n * sizeof(T), cudaMemcpyDeviceToDevice, st));
  int rc = std::is_same<T, double>::value
               ? rvvla_crs_spmv_f64(A, -1.0, reinterpret_cast<const double*>(x), 1.0, reinterpret_cast<double*>(r),
                                    (void*)st)
               : rvvla_crs_spmv_f32(A, -1.0f, reinterpret_cast<const float*>(x), 1.0f, reinterpret_cast<float*>(r),
                                    (void*)st);
  if (rc) return rc;
  RVVLA_CUDA(cudaMemcpyAsync(p, r, (size_t)n * sizeof(T), cudaMemcpyDeviceToDevice, st));
  cg_dot_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, r, r, rrp);
  RVVLA_LAUNCHED("cg_dot_kernel");
  cg_set_kernel<<<1, kRedThreads, 0, st>>>(rrp, upd_blocks, s, 0);
  RVVLA_LAUNCHED("cg_set_kernel");
  cg_dot_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, b, b, rrp);
  RVVLA_LAUNCHED("cg_dot_kernel");
  cg_set_kernel<<<1, kRedThreads, 0, st>>>(rrp, upd_blocks, s, 1);
  RVVLA_LAUNCHED("cg_set_kernel");
  CgScalars hs{};
  auto read_back = [&]() -> int {
    RVVLA_CUDA(cudaMemcpyAsync(&hs, s, sizeof(hs), cudaMemcpyDeviceToHost, st));
    RVVLA_CUDA(cudaStreamSynchronize(st));
    return RVVLA_OK;
  };
  if ((rc = read_back())) return rc;
  const double bb = hs.bb > 0.0 ? hs.bb : 1.0;
  int64_t it = 0;
  int cur = 0;
  bool done = std::sqrt(hs.rr[0] / bb) <= rtol;
  while (!done && it < max_iter) {
    rc = std::is_same<T, double>::value
             ? crs_spmv_dot_f64(A, reinterpret_cast<const double*>(p), reinterpret_cast<double*>(q), cd, st)
             : crs_spmv_dot_f32(A, reinterpret_cast<const float*>(p), reinterpret_cast<float*>(q), cd, st);
    if (rc) return rc;
    RVVLA_CHAIN(true, cg_update_kernel<T>, upd_blocks, kUpdThreads, st, n, r, q, s, cur, rrp);
    RVVLA_CHAIN(true, cg_xp_kernel<T>, (n + 255) / 256, 256, st, n, x, p, r, s, cur);
    cur ^= 1;
    ++it;
    if (it % check_every == 0 || it == max_iter) {
      if ((rc = read_back())) return rc;
      done = std::sqrt(hs.rr[cur] / bb) <= rtol;
    }
  }
  *iters = it;
  *rel_res = std::sqrt(hs.rr[cur] / bb);
  return RVVLA_OK;
}

// ---------------------------------------------------------------- BiCGStab
// Unpreconditioned BiCGStab (van der Vorst 1992) for a general square A, on
// the same pieces: per iteration two CRS products (v = A p, t = A s), the
// dots r^.v, t.s, t.t, r^.r and r.r as per-block partials summed by one
// block in a fixed order, and three fused vector passes.  Scalars stay on
// the device; the host reads them every check_every iterations.
struct BiScalars {
  double rho;    // r^.r of the current residual
  double alpha, omega, beta;
  double rr;     // r.r
  double bb;     // b.b
  int breakdown;  // rho, r^.v or t.t became exactly zero
};

template <class T>
__global__ void __launch_bounds__(kUpdThreads) bi_p_kernel(int64_t n, T* __restrict__ p, const T* __restrict__ r,
                                                           const T* __restrict__ v, const BiScalars* __restrict__ s) {
  const T beta = (T)s->beta, omega = (T)s->omega;
  for (int64_t i = (int64_t)blockIdx.x * kUpdThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kUpdThreads)
    p[i] = r[i] + beta * (p[i] - omega * v[i]);
}

__global__ void __launch_bounds__(kRedThreads) bi_alpha_kernel(const double* __restrict__ part, int64_t np,
                                                               BiScalars* s) {
  const double rv = block_sum(part, np);
  if (threadIdx.x == 0) {
    s->alpha = rv != 0.0 ? s->rho / rv : 0.0;
    if (rv == 0.0) s->breakdown = 1;
  }
}

template <class T>
__global__ void __launch_bounds__(kUpdThreads) bi_s_kernel(int64_t n, T* __restrict__ sv, const T* __restrict__ r,
                                                           const T* __restrict__ v, const BiScalars* __restrict__ s) {
  const T alpha = (T)s->alpha;
  for (int64_t i = (int64_t)blockIdx.x * kUpdThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kUpdThreads)
    sv[i] = r[i] - alpha * v[i];
}

// partials of u1.v1 and u2.v2 in one pass
template <class T>
__global__ void __launch_bounds__(kUpdThreads) dot2_kernel(int64_t n, const T* __restrict__ u1, const T* __restrict__ v1,
                                                           const T* __restrict__ u2, const T* __restrict__ v2,
                                                           double* __restrict__ part1, double* __restrict__ part2) {
  double a = 0.0, b = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kUpdThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kUpdThreads) {
    a += (double)u1[i] * (double)v1[i];
    b += (double)u2[i] * (double)v2[i];
  }
  block_partial(a, part1);
  block_partial(b, part2);
}

__global__ void __launch_bounds__(kRedThreads) bi_omega_kernel(const double* __restrict__ part1,
                                                               const double* __restrict__ part2, int64_t np,
                                                               BiScalars* s) {
  const double ts = block_sum(part1, np);
  __syncthreads();  // every thread has read the first sum before the second reuses the buffer
  const double tt = block_sum(part2, np);
  if (threadIdx.x == 0) {
    s->omega = tt != 0.0 ? ts / tt : 0.0;
    if (tt == 0.0) s->breakdown = 1;
  }
}

// x += alpha p + omega s, r = s - omega t, partials of r^.r and r.r
template <class T>
__global__ void __launch_bounds__(kUpdThreads) bi_xr_kernel(int64_t n, T* __restrict__ x, T* __restrict__ r,
                                                            const T* __restrict__ p, const T* __restrict__ sv,
                                                            const T* __restrict__ t, const T* __restrict__ rh,
                                                            const BiScalars* __restrict__ s, double* __restrict__ part1,
                                                            double* __restrict__ part2) {
  const T alpha = (T)s->alpha, omega = (T)s->omega;
  double a = 0.0, b = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kUpdThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kUpdThreads) {
    x[i] += alpha * p[i] + omega * sv[i];
    const T ri = sv[i] - omega * t[i];
    r[i] = ri;
    a += (double)rh[i] * (double)ri;
    b += (double)ri * (double)ri;
  }
  block_partial(a, part1);
  block_partial(b, part2);
}

__global__ void __launch_bounds__(kRedThreads) bi_rho_kernel(const double* __restrict__ part1,
                                                             const double* __restrict__ part2, int64_t np,
                                                             BiScalars* s, int init) {
  const double rho = block_sum(part1, np);
  __syncthreads();  // as above
  const double rr = block_sum(part2, np);
  if (threadIdx.x == 0) {
    if (init) {
      s->beta = 0.0;
      s->omega = 1.0;
      s->alpha = 1.0;
      s->breakdown = 0;
    } else {
      const bool ok = s->rho != 0.0 && s->omega != 0.0;
      s->beta = ok ? (rho / s->rho) * (s->alpha / s->omega) : 0.0;
      if (!ok || rho == 0.0) s->breakdown = 1;
    }
    s->rho = rho;
    s->rr = rr;
  }
}

template <class T>
int crs_product(const rvvla_crs* A, const T* x, T* y, cudaStream_t st) {
  return std::is_same<T, double>::value
             ? rvvla_crs_spmv_f64(A, 1.0, reinterpret_cast<const double*>(x), 0.0, reinterpret_cast<double*>(y),
                                  (void*)st)
             : rvvla_crs_spmv_f32(A, 1.0f, reinterpret_cast<const float*>(x), 0.0f, reinterpret_cast<float*>(y),
                                  (void*)st);
}

template <class T>
int bicgstab_impl(const rvvla_crs* A, const T* b, T* x, int64_t max_iter, double rtol, int64_t check_every,
                  int64_t* iters, double* rel_res, int* breakdown, cudaStream_t st) {
  if (!A || !b || !x || !iters || !rel_res || !breakdown) return fail(RVVLA_ERR_INVALID_ARG, "bicgstab: null argument");
  if (A->m != A->n || A->m <= 0) return fail(RVVLA_ERR_INVALID_ARG, "bicgstab: A must be square and non-empty");
  if (max_iter < 0 || check_every <= 0 || !(rtol >= 0.0))
    return fail(RVVLA_ERR_INVALID_ARG, "bicgstab: bad iteration limits");
  if (A->nz == 0 || !A->plan || (A->plan_kind != 1 && A->plan_kind != 2))
    return fail(RVVLA_ERR_INVALID_ARG, "bicgstab: A needs nonzeros and an analysed plan (rvvla_crs_analyze)");
  const int64_t n = A->n;
  const int upd_blocks = (int)std::min<int64_t>((n + kUpdThreads - 1) / kUpdThreads, (int64_t)sm_count() * 8);
  Scratch sc;
  const size_t vec = ((size_t)n * sizeof(T) + 255) / 256 * 256;
  const size_t pb = ((size_t)upd_blocks * sizeof(double) + 255) / 256 * 256;
  RVVLA_CUDA(sc.alloc_kept(6 * vec + 2 * pb + sizeof(BiScalars), st));
  char* base = sc.as<char>();
  T* r = reinterpret_cast<T*>(base);
  T* rh = reinterpret_cast<T*>(base + vec);
  T* p = reinterpret_cast<T*>(base + 2 * vec);
  T* v = reinterpret_cast<T*>(base + 3 * vec);
  T* sv = reinterpret_cast<T*>(base + 4 * vec);
  T* t = reinterpret_cast<T*>(base + 5 * vec);
  double* part1 = reinterpret_cast<double*>(base + 6 * vec);
  double* part2 = reinterpret_cast<double*>(base + 6 * vec + pb);
  BiScalars* s = reinterpret_cast<BiScalars*>(base + 6 * vec + 2 * pb);
  // r = b - A x, r^ = r, p = v = 0, rho = r^.r, b.b
  RVVLA_CUDA(cudaMemcpyAsync(r, b, (size_t)n * sizeof(T), cudaMemcpyDeviceToDevice, st));
  int rc = std::is_same<T, double>::value
               ? rvvla_crs_spmv_f64(A, -1.0, reinterpret_cast<const double*>(x), 1.0, reinterpret_cast<double*>(r),
                                    (void*)st)
               : rvvla_crs_spmv_f32(A, -1.0f, reinterpret_cast<const float*>(x), 1.0f, reinterpret_cast<float*>(r),
                                    (void*)st);
  if (rc) return rc;
  RVVLA_CUDA(cudaMemcpyAsync(rh, r, (size_t)n * sizeof(T), cudaMemcpyDeviceToDevice, st));
  RVVLA_CUDA(cudaMemsetAsync(p, 0, 2 * vec, st));  // p and v
  dot2_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, rh, r, r, r, part1, part2);
  RVVLA_LAUNCHED("dot2_kernel");
  bi_rho_kernel<<<1, kRedThreads, 0, st>>>(part1, part2, upd_blocks, s, 1);
  RVVLA_LAUNCHED("bi_rho_kernel");
  cg_dot_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, b, b, part1);
  RVVLA_LAUNCHED("cg_dot_kernel");
  sum_to_kernel<double><<<1, kRedThreads, 0, st>>>(part1, upd_blocks, &s->bb);
  RVVLA_LAUNCHED("sum_to_kernel");
  BiScalars hs{};
  auto read_back = [&]() -> int {
    RVVLA_CUDA(cudaMemcpyAsync(&hs, s, sizeof(hs), cudaMemcpyDeviceToHost, st));
    RVVLA_CUDA(cudaStreamSynchronize(st));
    return RVVLA_OK;
  };
  if ((rc = read_back())) return rc;
  const double bb = hs.bb > 0.0 ? hs.bb : 1.0;
  int64_t it = 0;
  bool done = std::sqrt(hs.rr / bb) <= rtol;
  while (!done && it < max_iter) {
    bi_p_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, p, r, v, s);
    RVVLA_LAUNCHED("bi_p_kernel");
    if ((rc = crs_product<T>(A, p, v, st))) return rc;
    cg_dot_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, rh, v, part1);
    RVVLA_LAUNCHED("cg_dot_kernel");
    bi_alpha_kernel<<<1, kRedThreads, 0, st>>>(part1, upd_blocks, s);
    RVVLA_LAUNCHED("bi_alpha_kernel");
    bi_s_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, sv, r, v, s);
    RVVLA_LAUNCHED("bi_s_kernel");
    if ((rc = crs_product<T>(A, sv, t, st))) return rc;
    dot2_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, t, sv, t, t, part1, part2);
    RVVLA_LAUNCHED("dot2_kernel");
    bi_omega_kernel<<<1, kRedThreads, 0, st>>>(part1, part2, upd_blocks, s);
    RVVLA_LAUNCHED("bi_omega_kernel");
    bi_xr_kernel<T><<<upd_blocks, kUpdThreads, 0, st>>>(n, x, r, p, sv, t, rh, s, part1, part2);
    RVVLA_LAUNCHED("bi_xr_kernel");
    bi_rho_kernel<<<1, kRedThreads, 0, st>>>(part1, part2, upd_blocks, s, 0);
    RVVLA_LAUNCHED("bi_rho_kernel");
    ++it;
    if (it % check_every == 0 || it == max_iter) {
      if ((rc = read_back())) return rc;
      done = std::sqrt(hs.rr / bb) <= rtol || hs.breakdown;
    }
  }
  *iters = it;
  *rel_res = std::sqrt(hs.rr / bb);
  *breakdown = hs.breakdown && !(std::sqrt(hs.rr / bb) <= rtol);
  return RVVLA_OK;
}

}  // namespace
}  // namespace rvvla

using namespace rvvla;

extern "C" {

int rvvla_cg_f64(const rvvla_crs* A, const double* b, double* x, int64_t max_iter, double rtol, int64_t check_every,
                 int64_t* iters, double* rel_res, void* stream) {
  return cg_impl<double>(A, b, x, max_iter, rtol, check_every, iters, rel_res, as_stream(stream));
}

int rvvla_cg_f32(const rvvla_crs* A, const float* b, float* x, int64_t max_iter, double rtol, int64_t check_every,
                 int64_t* iters, double* rel_res, void* stream) {
  return cg_impl<float>(A, b, x, max_iter, rtol, check_every, iters, rel_res, as_stream(stream));
}

int rvvla_bicgstab_f64(const rvvla_crs* A, const double* b, double* x, int64_t max_iter, double rtol,
                       int64_t check_every, int64_t* iters, double* rel_res, int* breakdown, void* stream) {
  return bicgstab_impl<double>(A, b, x, max_iter, rtol, check_every, iters, rel_res, breakdown, as_stream(stream));
}

int rvvla_bicgstab_f32(const rvvla_crs* A, const float* b, float* x, int64_t max_iter, double rtol,
                       int64_t check_every, int64_t* iters, double* rel_res, int* breakdown, void* stream) {
  return bicgstab_impl<float>(A, b, x, max_iter, rtol, check_every, iters, rel_res, breakdown, as_stream(stream));
}

int rvvla_crs_spmv_dot_f64(const rvvla_crs* A, const double* x, double* y, double* dot, void* stream) {
  return spmv_dot_impl<double>(A, x, y, dot, as_stream(stream));
}

int rvvla_crs_spmv_dot_f32(const rvvla_crs* A, const float* x, float* y, float* dot, void* stream) {
  return spmv_dot_impl<float>(A, x, y, dot, as_stream(stream));
}

}  // extern "C"
