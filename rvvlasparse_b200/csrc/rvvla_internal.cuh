// rvvla_internal.cuh — shared pieces of the sm_100a kernels and the C ABI:
// status plumbing, stream-ordered scratch, cache-policy loads, warp scans.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <atomic>
#include <string>

#include "rvvla.h"

namespace rvvla {

// ------------------------------------------------------------------ status
void set_error(const std::string& msg);
int fail(int status, const std::string& msg);
int cuda_fail(cudaError_t e, const char* where);
void count_launch(uint64_t n = 1);

#define RVVLA_CUDA(call)                                      \
  do {                                                        \
    cudaError_t e_ = (call);                                  \
    if (e_ != cudaSuccess) return ::rvvla::cuda_fail(e_, #call); \
  } while (0)

// Checks the launch that just happened and counts it.
#define RVVLA_LAUNCHED(name)                                         \
  do {                                                               \
    cudaError_t e_ = cudaGetLastError();                             \
    if (e_ != cudaSuccess) return ::rvvla::cuda_fail(e_, name);      \
    ::rvvla::count_launch();                                         \
  } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

int sm_count();
// Per-device status word set by kernels whose bounded waits expired.
int* device_status_word();

// Ask for the largest shared-memory carveout for a kernel whose occupancy is
// bounded by its shared memory (set once per kernel instantiation).
template <class K>
inline void prefer_shared(K kernel) {
  static std::atomic<bool> done{false};
  if (!done.load(std::memory_order_relaxed)) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    cudaGetLastError();
    done.store(true, std::memory_order_relaxed);
  }
}

// The current device's pool for temporary buffers, made on first use; null if
// it could not be made.
cudaMemPool_t scratch_pool();
// Gives back what that pool keeps unused; false if there is none or it fails.
bool trim_scratch_pool();

// A launch chained to the stream's previous kernel if `chained`.
#define RVVLA_CHAIN(chained, kernel, blocks, threads, st, ...)                                        \
  do {                                                                                                \
    RVVLA_CUDA(::rvvla::launch_chained(kernel, (unsigned)(blocks), threads, chained, st, __VA_ARGS__)); \
    ::rvvla::count_launch();                                                                          \
  } while (0)

// Stream-ordered temporary buffer.  alloc() takes it from the device's default
// pool (builders, and the ordinary fp64 CSR5 product, whose callers account
// for that pool).  alloc_kept() is for products: it takes up to kScratchKeep
// bytes from the library's own pool, which keeps that much when a stream is
// synchronised; the default pool keeps nothing, so the first product after a
// synchronisation mapped its few KB of carries anew (the CRS fp64 product of
// 4M power-law rows, first call on a new matrix: 883 us, 406 us with the kept
// pool; a first CG solve on 4M rows 8.7 -> 6.0 ms).  Builders stay away from
// it: the LAV builder's buffers, trimmed to the limit at each of its
// synchronisations, took 118 ms instead of 31; the SELL builder takes its
// buffers there where they are small (a batch's matrices).
constexpr uint64_t kScratchKeep = 256ull << 20;  // a solve on 8M rows in fp64 fits
struct Scratch {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  cudaError_t alloc(size_t bytes, cudaStream_t st) {
    s = st;
    cudaError_t e = cudaMallocAsync(&p, bytes == 0 ? 16 : bytes, st);
    if (e == cudaErrorMemoryAllocation && trim_scratch_pool()) {  // without what the library's pool keeps
      cudaGetLastError();
      e = cudaMallocAsync(&p, bytes == 0 ? 16 : bytes, st);
    }
    return e;
  }
  cudaError_t alloc_kept(size_t bytes, cudaStream_t st) {
    cudaMemPool_t pool = bytes <= kScratchKeep ? scratch_pool() : nullptr;
    if (!pool) return alloc(bytes, st);
    s = st;
    const cudaError_t e = cudaMallocFromPoolAsync(&p, bytes == 0 ? 16 : bytes, pool, st);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    return alloc(bytes, st);
  }
  ~Scratch() {
    if (p) cudaFreeAsync(p, s);
  }
  template <class T>
  T* as() const { return reinterpret_cast<T*>(p); }
};

// Buffers of the CRS product with a fused dot (crs.cu; the solvers').  part:
// one entry of the value type per warp, sums: one double per 128 warps,
// ticket: 0 before and after a product, out: the dot.
struct CrsDot {
  void* part;
  double* sums;
  unsigned* ticket;
  double* out;
};

// Launches that may start while the stream's previous kernel drains: the
// kernel calls grid_chain() (or chain_wait() later) before it touches anything
// the kernels before it write or read.  In a chain of short kernels this hides
// launches and ramp-ups.  The first kernel of a call is launched the ordinary
// way, so that whatever the caller enqueued before is complete.
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), unsigned blocks, unsigned threads, bool chained, cudaStream_t st,
                                  A... args) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = chained ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// What the kernels before it in the chain write, a chained kernel reads through
// ordinary loads from pointers without __restrict__, or ld_chain: ld.global.nc
// and a restrict argument promise data that nothing writes while the kernel
// runs, and it runs from before its wait on, so that either may be read early.
//
// By every CTA that does any work: chain_open lets the stream's next chained
// kernel start once all CTAs have come here, chain_wait waits until the
// previous kernel is complete and its writes are visible (at once in a kernel
// launched the ordinary way).
__device__ __forceinline__ void chain_open() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_chain() {
  chain_open();
  chain_wait();
}

// ------------------------------------------------------------------ loads
// Streaming operands (values, indices) are read once: evict-first in L2 and
// no L1 allocation.  The gathered vector x is re-read across the whole matrix:
// evict-last keeps it resident in the 126 MB L2.  The asm statements are not
// volatile: they are pure reads of data that neither the kernel nor one that it
// is chained to writes, so the compiler may hoist and batch them to keep many
// loads in flight.
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

template <class T> __device__ __forceinline__ T ld_stream(const T* p, uint64_t pol);
template <> __device__ __forceinline__ double ld_stream<double>(const double* p, uint64_t pol) {
  double v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ float ld_stream<float>(const float* p, uint64_t pol) {
  float v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ int ld_stream<int>(const int* p, uint64_t pol) {
  int v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ unsigned ld_stream<unsigned>(const unsigned* p, uint64_t pol) {
  unsigned v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ unsigned short ld_stream<unsigned short>(const unsigned short* p, uint64_t pol) {
  unsigned short v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ __nv_bfloat16 ld_stream<__nv_bfloat16>(const __nv_bfloat16* p, uint64_t pol) {
  unsigned short v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
  return __ushort_as_bfloat16(v);
}
__device__ __forceinline__ int4 ld_stream_v4(const int4* p, uint64_t pol) {
  int4 v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.b32 {%0,%1,%2,%3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p), "l"(pol));
  return v;
}

template <class T> __device__ __forceinline__ T ld_keep(const T* p, uint64_t pol);
template <> __device__ __forceinline__ double ld_keep<double>(const double* p, uint64_t pol) {
  double v;
  asm("ld.global.nc.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
template <> __device__ __forceinline__ float ld_keep<float>(const float* p, uint64_t pol) {
  float v;
  asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}

// The gathered vector where the kernel before in the chain wrote it (see
// launch_chained): a coherent load that stays behind the wait.
__device__ __forceinline__ double ld_chain(const double* p, uint64_t pol) {
  double v;
  asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol) : "memory");
  return v;
}
__device__ __forceinline__ float ld_chain(const float* p, uint64_t pol) {
  float v;
  asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol) : "memory");
  return v;
}

// value conversion for mixed storage
template <class V> __device__ __forceinline__ float to_f32(V v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// ------------------------------------------------------------------ two-sum
// Compensated fp32 accumulation (Knuth's TwoSum): s + c carries the running
// sum with the rounding error of every addition kept in c.
struct CompF32 {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    float t = s + v;
    float bp = t - s;
    float err = (s - (t - bp)) + (v - bp);
    s = t;
    c += err;
  }
  __device__ __forceinline__ void add(const CompF32& o) {
    add(o.s);
    c += o.c;
  }
  __device__ __forceinline__ float value() const { return s + c; }
};

// ------------------------------------------------------------------ warp scan
// Inclusive segmented sum over the warp: lanes with head=true start a new
// segment.  Works for any type with operator+.
template <class T>
__device__ __forceinline__ T warp_seg_scan(T v, bool head, unsigned lane) {
  unsigned heads = __ballot_sync(0xffffffffu, head);
  // distance to the segment's first lane
  unsigned below = heads & ((2u << lane) - 1u);  // heads at lanes <= lane
  int seg_start = below ? (31 - __clz(below)) : 0;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    T o = __shfl_up_sync(0xffffffffu, v, d);
    if ((int)lane - d >= seg_start) v = v + o;
  }
  return v;
}

}  // namespace rvvla
