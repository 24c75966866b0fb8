// Shared helpers for the sm_103a kernels of libbilu_isai.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "bilu_isai.h"
#include "perdevice.cuh"

namespace bilu {

// Last CUDA error seen by a host entry point of this thread.
extern thread_local int g_last_cuda_error;
// Kernel launches issued by this library (all threads), for accounting.
extern unsigned long long g_launches;

inline int cuda_status(cudaError_t e) {
  if (e == cudaSuccess) return BILU_OK;
  g_last_cuda_error = (int)e;
  return BILU_ERR_CUDA;
}

#define BILU_TRY_CUDA(call)                          \
  do {                                               \
    cudaError_t e_ = (call);                         \
    if (e_ != cudaSuccess) return ::bilu::cuda_status(e_); \
  } while (0)

#define BILU_TRY(call)               \
  do {                               \
    int st_ = (call);                \
    if (st_ != BILU_OK) return st_;  \
  } while (0)

#define BILU_LAUNCH_CHECK()                                    \
  do {                                                         \
    __atomic_fetch_add(&::bilu::g_launches, 1ull, __ATOMIC_RELAXED); \
    BILU_TRY_CUDA(cudaGetLastError());                         \
  } while (0)

inline cudaStream_t S(bilu_stream_t s) { return (cudaStream_t)s; }

inline bool bs_supported(int bs) { return bs == 4 || bs == 5 || bs == 8; }

// Dispatch a templated launcher over the built block sizes.
#define BILU_DISPATCH_BS(bs, FN, ...)                 \
  ((bs) == 4   ? FN<4>(__VA_ARGS__)                    \
   : (bs) == 5 ? FN<5>(__VA_ARGS__)                    \
   : (bs) == 8 ? FN<8>(__VA_ARGS__)                    \
               : BILU_ERR_UNSUPPORTED)

inline unsigned ceil_div(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

// The current device's value in c (PerDevice::get).
template <class V, class F>
int per_device(PerDevice<V>& c, V* out, F make) {
  int dev = 0;
  BILU_TRY_CUDA(cudaGetDevice(&dev));
  return c.get(dev, out, make);
}

// Dynamic shared memory above 48 KB for fn, allowed once per device.
inline int allow_smem(PerDevice<int>& c, const void* fn, size_t bytes) {
  int ok = 0;
  return per_device(c, &ok, [&](int*) -> int {
    BILU_TRY_CUDA(
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return BILU_OK;
  });
}

// Workspace carving: aligned sub-allocations from a caller buffer.
struct Carver {
  char* base;
  size_t cap, used;
  Carver(void* p, size_t n) : base((char*)p), cap(n), used(0) {}
  template <class T>
  T* take(size_t count) {
    size_t off = (used + 255) & ~(size_t)255;
    size_t need = off + count * sizeof(T);
    if (need > cap || (base == nullptr && count > 0)) return nullptr;
    used = need;
    return (T*)(base + off);
  }
};
inline size_t carve_size(size_t bytes) { return ((bytes + 255) & ~(size_t)255) + 256; }

// ---------------------------------------------------------------- device
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <class T>
__device__ __forceinline__ T warp_sum(T v, unsigned mask = 0xffffffffu) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}

// Programmatic dependent launch (k_bsr_spmv, DEP): the launch before this one
// in the stream has finished and its writes are visible / the next one may start.
__device__ __forceinline__ void dependency_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void dependents_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Streaming (evict-first) loads for values read exactly once.
__device__ __forceinline__ double2 ld_stream(const double2* p) {
  double2 v;
  asm volatile("ld.global.cs.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_stream(const float4* p) {
  float4 v;
  asm volatile("ld.global.cs.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_stream(const double* p) {
  double v;
  asm volatile("ld.global.cs.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
  float v;
  asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// The bits of a double (hi, lo) whose rounding to FP32 is a normal number or
// infinity, rounded.
__device__ __forceinline__ float narrow_normal(unsigned hi, unsigned lo) {
  // nine exponent bits and the first 23 of the fraction; the exponents in
  // question, 897 to 1150, differ from FP32's by 384 modulo 512
  const unsigned m = __funnelshift_l(lo, hi, 3);
  // the 29 bits left over against one half, ties to even (a carry may run into
  // the exponent, up to infinity)
  const unsigned up = ((lo << 3) | (m & 1u)) > 0x80000000u ? 1u : 0u;
  return __uint_as_float((m - (384u << 23) + up) | (hi & 0x80000000u));
}

// double -> float, round to nearest even, on the integer pipe: the same bits as
// the conversion instruction, which runs at the FP64 rate on GB300 (64 cycles a
// warp instruction per SM sub-partition against about 9 for this).  A value
// whose result is neither zero nor a normal float (subnormal, overflow, NaN)
// takes the instruction.
__device__ __forceinline__ float narrow(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  if ((hi & 0x7fffffffu) - (897u << 20) >= (254u << 20)) {
    if (((hi << 1) | lo) == 0) return __uint_as_float(hi);
    return __double2float_rn(d);
  }
  return narrow_normal(hi, lo);
}

// narrow() of N values with one branch for all of them.
template <int N>
__device__ __forceinline__ void narrow_all(const double (&d)[N], float (&f)[N]) {
  unsigned worst = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const unsigned hi = (unsigned)__double2hiint(d[i]), lo = (unsigned)__double2loint(d[i]);
    worst = max(worst, (hi & 0x7fffffffu) - (897u << 20));
    f[i] = narrow_normal(hi, lo);
  }
  if (worst >= (254u << 20)) {
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = narrow(d[i]);
  }
}

// float -> double (exact), likewise on the integer pipe.
__device__ __forceinline__ double widen(float f) {
  const unsigned u = __float_as_uint(f), a = u & 0x7fffffffu;
  if (a - 0x00800000u >= 0x7f000000u) {  // zero, subnormal, infinity, NaN
    if (a == 0) return __hiloint2double((int)u, 0);
    return (double)f;
  }
  return __hiloint2double((int)((u & 0x80000000u) | ((a >> 3) + (896u << 20))), (int)(u << 29));
}

// Rows of a product with more blocks than this are long: power-law hub rows hold
// up to ~2000, and a lane group alone runs one dependent FMA chain over all of
// them while the rest of the GPU idles.
constexpr int kLongSpmvRow = 64;

// The entries [s, e) of a pattern row per thread, f(row, p) for each: a thread
// walks its own row, except that rows of more than kSharedRow entries are
// walked by the whole warp, 32 entries at a time (one thread alone takes
// hundreds of microseconds over a power-law hub row of 2000 entries with an
// atomic each, while the rest of the GPU idles).  Called by all 32 lanes;
// threads without a row pass s = e.
constexpr int kSharedRow = 48;
template <class F>
__device__ __forceinline__ void for_row_entries(int row, int s, int e, F f) {
  const bool shared = e - s > kSharedRow;
  if (!shared)
    for (int p = s; p < e; ++p) f(row, p);
  unsigned todo = __ballot_sync(0xffffffffu, shared);
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    const int r = __shfl_sync(0xffffffffu, row, src);
    const int a = __shfl_sync(0xffffffffu, s, src), b = __shfl_sync(0xffffffffu, e, src);
    for (int p = a + (int)(threadIdx.x & 31); p < b; p += 32) f(r, p);
  }
}

// Bounded spin budget for sync-free kernels: after this many polls of a
// dependency flag the waiter records BILU_ERR_TIMEOUT and returns.
// Polls back off up to 256 ns, so the budget bounds a wait at a few seconds.
constexpr long long kSpinLimit = 1ll << 22;

// Caller-owned home for the level analysis of the lower DAG that BILU(0)
// computes (order[nb+1], lvl_ptr[nb+2], nlev[4]), so that lower triangular
// solves on the factor can reuse it; the host words are filled on return.
struct LevelOut {
  int *order = nullptr, *lvl = nullptr, *nlev = nullptr;
  int h_nlev = 0, h_sched = 0, h_maxdeg = 0;  // levels, solve schedule, largest dependency count
  int h_fsched = 0;                           // recommended factorisation schedule
  // optional match lists of BILU(0)'s updates (bilu0_match_count / _fill):
  // positions mptr[p] .. mptr[p+1] of mpair for block position p
  const int* mptr = nullptr;
  const int2* mpair = nullptr;
  // BILU(0)'s plan, one entry per stored block (k_bilu0_plan), and whether the
  // pattern takes the row flow
  int2* plan = nullptr;
  int h_rowflow = 0;
  int h_blocks = 0;   // long rows hold enough to take the factorisation by blocks
  int h_counted = 0;  // the caller's block count covers the stored blocks
  // test hook: polls before a wait of the factorisation gives up, and a row that
  // never publishes (-1: none)
  long long spin = kSpinLimit;
  int withhold = -1;
};

}  // namespace bilu
