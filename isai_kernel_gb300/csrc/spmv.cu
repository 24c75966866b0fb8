// BSR SpMV / SpMM and the ISAI preconditioner apply (sm_103a).
//
// Replaces bcsr_spmv (bcsc2bcsrAndSpMV.h:49, thread per block row, scalar
// loops) and the DMMA variants of bsr_tensor_SpMV.h:21-400.  On GB300 the FP64
// pipe (measured 1.2 TFLOP/s DFMA, 1.05 TFLOP/s DMMA m8n8k4) is the binding
// limit of an FP64 BSR SpMV (1 DFMA per 8 B of values), so the layout spends
// FP64 instructions only on the block products: one lane per scalar row
// accumulates across every block of its block row and needs no reduction.
// The bs lanes of a block row read the bs rows of each block, so every block
// (bs*bs*8 bytes) is fetched in whole 32-byte sectors by one group, and the x
// segment is a broadcast within the group.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include <cooperative_groups.h>

#include "common.cuh"

namespace bilu {

namespace {

template <class T>
struct Vec;
template <>
struct Vec<double> {
  static constexpr int W = 2;
  using V = double2;
};
template <>
struct Vec<float> {
  static constexpr int W = 4;
  using V = float4;
};

__device__ __forceinline__ double to_acc(double v, double) { return v; }
__device__ __forceinline__ double to_acc(float v, double) { return (double)v; }
__device__ __forceinline__ float to_acc(double v, float) { return (float)v; }
__device__ __forceinline__ float to_acc(float v, float) { return v; }

// Reads of x where the launch before may still have been writing it when this
// one started: not the read-only path.  They cannot move above dependency_wait
// because the pointer comes out of after_wait.
template <class T>
__device__ __forceinline__ const T* after_wait(const T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}
__device__ __forceinline__ double ld_dep(const double* p) {
  double v;
  asm("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_dep(const float* p) {
  float v;
  asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld_dep(const double2* p) {
  double2 v;
  asm("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_dep(const float4* p) {
  float4 v;
  asm("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p));
  return v;
}
template <bool DEP, class T>
__device__ __forceinline__ T ld_x(const T* p) {
  if constexpr (DEP) return ld_dep(p);
  else return __ldg(p);
}

// Load the BS-long x segment of block column bc into registers (AccT).
template <int BS, class XT, class AccT, bool DEP = false>
__device__ __forceinline__ void load_x(const XT* x, long long bc, AccT* xr) {
  const XT* p = x + bc * BS;
  constexpr int W = Vec<XT>::W;
  if constexpr (BS % W == 0) {
    // the segment starts at bc*BS elements: 16-byte aligned when BS is a
    // multiple of the vector width
    using V = typename Vec<XT>::V;
#pragma unroll
    for (int c = 0; c < BS / W; ++c) {
      V v = ld_x<DEP>(reinterpret_cast<const V*>(p) + c);
      if constexpr (W == 2) {
        xr[2 * c] = to_acc(v.x, AccT());
        xr[2 * c + 1] = to_acc(v.y, AccT());
      } else {
        xr[4 * c] = to_acc(v.x, AccT());
        xr[4 * c + 1] = to_acc(v.y, AccT());
        xr[4 * c + 2] = to_acc(v.z, AccT());
        xr[4 * c + 3] = to_acc(v.w, AccT());
      }
    }
  } else {
#pragma unroll
    for (int c = 0; c < BS; ++c) xr[c] = to_acc(ld_x<DEP>(p + c), AccT());
  }
}

// Row r of block p (BS values) into registers, streaming loads.
template <int BS, class VT, class AccT>
__device__ __forceinline__ void load_row(const VT* __restrict__ val, long long p, int r, AccT* a) {
  const VT* q = val + (p * BS + r) * BS;
  constexpr int W = Vec<VT>::W;
  if constexpr (BS % W == 0) {
    using V = typename Vec<VT>::V;
#pragma unroll
    for (int c = 0; c < BS / W; ++c) {
      V v = ld_stream(reinterpret_cast<const V*>(q) + c);
      if constexpr (W == 2) {
        a[2 * c] = to_acc(v.x, AccT());
        a[2 * c + 1] = to_acc(v.y, AccT());
      } else {
        a[4 * c] = to_acc(v.x, AccT());
        a[4 * c + 1] = to_acc(v.y, AccT());
        a[4 * c + 2] = to_acc(v.z, AccT());
        a[4 * c + 3] = to_acc(v.w, AccT());
      }
    }
  } else {
#pragma unroll
    for (int c = 0; c < BS; ++c) a[c] = to_acc(ld_stream(q + c), AccT());
  }
}

// Row r of the transpose of block p: its column r.  The BS lanes of a block row
// read neighbouring columns, so each of the BS loads is one run of BS values.
template <int BS, class VT, class AccT>
__device__ __forceinline__ void load_col(const VT* __restrict__ val, long long p, int r, AccT* a) {
  const VT* q = val + p * BS * BS + r;
#pragma unroll
  for (int c = 0; c < BS; ++c) a[c] = to_acc(__ldg(q + c * BS), AccT());
}

// Row r of entry p of the matrix: TR reads the transpose of block src[p] of
// another matrix's values (the transposed product, without transposing them).
template <int BS, bool TR, class VT, class AccT>
__device__ __forceinline__ void load_entry(const VT* __restrict__ val,
                                           const int* __restrict__ src, long long p, int r,
                                           AccT* a) {
  if constexpr (TR)
    load_col<BS, VT, AccT>(val, __ldg(src + p), r, a);
  else
    load_row<BS, VT, AccT>(val, p, r, a);
}

// The CTA's long rows (nslot slots, -1 for none): its NG groups
// take the blocks g, g + NG, ... of each (two accumulators, even and odd
// turns), the NG partials are added in group order.  Out of line so that
// the short rows' loop keeps its registers.  Called by every thread.
template <int BS, class VT, class XT, class YT, class AccT, int NG>
__device__ __noinline__ void spmv_long_rows(const int* long_rows, int nslot, const int* __restrict__ row,
                                            const int* __restrict__ col,
                                            const VT* __restrict__ val,
                                            const XT* __restrict__ x, YT* __restrict__ y,
                                            float* __restrict__ y32, AccT* red, bool in_group,
                                            int cg, int r) {
  for (int i = 0; i < nslot; ++i) {
    const int br = long_rows[i];
    if (br < 0) continue;  // uniform across the CTA (shared memory)
    const int rs = __ldg(row + br), re = __ldg(row + br + 1);
    AccT a0 = 0, a1 = 0;
    if (in_group) {
      int p = rs + cg;
      // F blocks' loads in flight; even turns go to a0, odd ones to a1
      auto turns = [&](auto f) {
        constexpr int F = decltype(f)::value;
        for (; p + (F - 1) * NG < re; p += F * NG) {
          AccT v[F][BS], xv[F][BS];
#pragma unroll
          for (int t = 0; t < F; ++t) load_row<BS, VT, AccT>(val, p + t * NG, r, v[t]);
#pragma unroll
          for (int t = 0; t < F; ++t) load_x<BS, XT, AccT>(x, __ldg(col + p + t * NG), xv[t]);
#pragma unroll
          for (int t = 0; t < F; t += 2)
#pragma unroll
            for (int k = 0; k < BS; ++k) {
              a0 = fma(v[t][k], xv[t][k], a0);
              a1 = fma(v[t + 1][k], xv[t + 1][k], a1);
            }
        }
      };
      turns(std::integral_constant<int, 4>());
      turns(std::integral_constant<int, 2>());
      if (p < re) {
        AccT v0[BS], x0[BS];
        load_row<BS, VT, AccT>(val, p, r, v0);
        load_x<BS, XT, AccT>(x, __ldg(col + p), x0);
#pragma unroll
        for (int k = 0; k < BS; ++k) a0 = fma(v0[k], x0[k], a0);
      }
      red[cg * BS + r] = a0 + a1;
    }
    __syncthreads();
    if (threadIdx.x < BS) {
      AccT t = 0;
      for (int q = 0; q < NG; ++q) t += red[q * BS + threadIdx.x];
      y[(long long)br * BS + threadIdx.x] = (YT)t;
      if (y32) y32[(long long)br * BS + threadIdx.x] = (float)t;
    }
    __syncthreads();
  }
}

// y = M x: lane group of BS lanes per block row, lane r owns scalar row r.
// FP64: bound by the FP64 pipe, where an instruction takes as long with lanes
// off, and as long predicated off.  So a warp's groups take one block each a turn
// and go on together until the longest row ends: no place past a row's end that
// all the groups have reached is issued, and the warps of a full SM cover the
// latency (two rows a group of the 4- and 5-blocks, two blocks a batch of the
// 8-blocks before; the apply, before -> now: 64^3 7-point 4x4 67.8 -> 63.7 us,
// 47x43x41 5x5 41.3 -> 38.9, 512^2 5-point 5x5 81.8 -> 77.9, 8x8 249 -> 172, 161
// of them DFMA at 1.25 TFLOP/s).
// FP32: bound by memory.  A group handles RPG consecutive block rows and issues
// the loads of the next U blocks of all of them before any arithmetic, so a warp
// keeps RPG*U independent block loads per lane in flight; each row's sum runs in
// block order whatever U and RPG are (the same bits).  Chosen by launch_spmv from
// measurements on the 128^3 7-point pattern (7 blocks a row) and its triangle (4
// a row): U = 4 with RPG = 1 for wider rows (0.199 -> 0.176 ms on the operator),
// RPG = 1 at 8 CTAs per SM for bs 4 rows of ~4 blocks, else RPG = 2.
// Patterns with rows of more than kLongSpmvRow blocks take k_bsr_spmv_balanced
// (FP64) or k_bsr_spmv_uneven (FP32), unless the rows are alike or the long ones
// few (launch_spmv); HUBS leaves those few to k_spmv_hubs.
// DEP, for a product whose x is the result of the launch before it (U after L,
// A after U): started by programmatic dependent launch while that one drains,
// it reads its row pointers, columns and first blocks, none of which the launch
// before writes, and waits before its first read of x and before any write.
// The launch before must itself have been ordered after whatever wrote the
// matrix.  It hides the tail of one product and the three dependent DRAM
// latencies at the start of the next (64^3 7-point, 4x4 blocks, the FP32 apply
// 33.7 -> 28.9 us, FP64 71.2 -> 67.9; 128^3 FP32 249 -> 224).
template <int BS, class VT, class XT, class YT, class AccT, int RPG, int U, int MINB, bool TR,
          bool DEP, bool HUBS>
__global__ void __launch_bounds__(256, MINB) k_bsr_spmv(int mb, const int* __restrict__ row,
                                                     const int* __restrict__ col,
                                                     const int* __restrict__ src,
                                                     const VT* __restrict__ val,
                                                     const XT* __restrict__ x,
                                                     YT* __restrict__ y,
                                                     float* __restrict__ y32) {
  constexpr int G = 32 / BS;  // lane groups per warp
  dependents_launch();
  int lane = threadIdx.x & 31;
  int g = lane / BS, r = lane - g * BS;
  long long base = (((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * G + g) * RPG;
  const unsigned live = __ballot_sync(0xffffffffu, g < G && base < mb);
  if (g >= G || base >= mb) return;
  int s[RPG], e[RPG];
  bool skip[RPG];
#pragma unroll
  for (int q = 0; q < RPG; ++q) {
    bool ok = base + q < mb;
    s[q] = ok ? __ldg(row + base + q) : 0;
    e[q] = ok ? __ldg(row + base + q + 1) : 0;
    skip[q] = HUBS && e[q] - s[q] > kLongSpmvRow;
    if (skip[q]) e[q] = s[q];
  }
  AccT acc[RPG];
#pragma unroll
  for (int q = 0; q < RPG; ++q) acc[q] = 0;
  const XT* xp = x;
  if constexpr (sizeof(AccT) == 8) {
    // one block at a time, the warp's groups together until the longest row ends
    static_assert(RPG == 1 && U == 1);
    int c = s[0] < e[0] ? __ldg(col + s[0]) : -1;
    for (int p = s[0]; __any_sync(live, p < e[0]); ++p) {
      AccT a[BS], xv[BS];
      if (c >= 0) load_entry<BS, TR, VT, AccT>(val, src, p, r, a);
      const int next = p + 1 < e[0] ? __ldg(col + p + 1) : -1;
      if constexpr (DEP) {
        if (p == s[0]) {
          dependency_wait();
          xp = after_wait(x);
        }
      }
      if (c >= 0) {
        load_x<BS, XT, AccT, DEP>(xp, c, xv);
#pragma unroll
        for (int k = 0; k < BS; ++k) acc[0] = fma(a[k], xv[k], acc[0]);
      }
      c = next;
    }
  } else {
    // batches of U blocks per row; every load of a batch (column indices,
    // block rows, x segments) is issued before its FMAs
    for (int off = 0;; off += U) {
      bool any = false;
#pragma unroll
      for (int q = 0; q < RPG; ++q) any |= s[q] + off < e[q];
      if (!any) break;
      int c[RPG][U];
#pragma unroll
      for (int q = 0; q < RPG; ++q)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          int p = s[q] + off + u;
          c[q][u] = p < e[q] ? __ldg(col + p) : -1;
        }
      AccT a[RPG][U][BS], xv[RPG][U][BS];
#pragma unroll
      for (int q = 0; q < RPG; ++q)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          // DEP: not on c, so that both loads go out before the wait
          if (DEP ? s[q] + off + u < e[q] : c[q][u] >= 0) {
            load_entry<BS, TR, VT, AccT>(val, src, s[q] + off + u, r, a[q][u]);
          } else {
#pragma unroll
            for (int k = 0; k < BS; ++k) a[q][u][k] = 0;
          }
        }
      if constexpr (DEP) {  // the first blocks wait in registers
        if (off == 0) {
          dependency_wait();
          xp = after_wait(x);
        }
      }
      // x segments (mostly L2 hits) are consumed as they arrive, which keeps
      // the register footprint low enough for 4 CTAs per SM with FP32 values
#pragma unroll
      for (int q = 0; q < RPG; ++q)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (c[q][u] >= 0) {
            load_x<BS, XT, AccT, DEP>(xp, c[q][u], xv[q][u]);
#pragma unroll
            for (int k = 0; k < BS; ++k) acc[q] = fma(a[q][u][k], xv[q][u][k], acc[q]);
          }
        }
    }
  }
  if constexpr (DEP) dependency_wait();  // rows without blocks
#pragma unroll
  for (int q = 0; q < RPG; ++q)
    if (base + q < mb && !skip[q]) {
      y[(base + q) * BS + r] = (YT)acc[q];
      if (y32) y32[(base + q) * BS + r] = (float)acc[q];  // optional FP32 copy
    }
}

// The long rows of a product whose other rows are short and alike (k_bsr_spmv, HUBS,
// leaves them out): a CTA each, its lane groups sharing the row's blocks.  The CTAs
// look for them CH rows at a time.  Started by programmatic dependent launch beside
// the other rows' kernel, it ends after that one (spmv_layout_word: when, and the
// times).
template <int BS, class VT, class XT, class YT>
__global__ void __launch_bounds__(256) k_spmv_hubs(int mb, int ch, const int* __restrict__ row,
                                                   const int* __restrict__ col,
                                                   const VT* __restrict__ val,
                                                   const XT* __restrict__ x, YT* __restrict__ y,
                                                   float* __restrict__ y32) {
  constexpr int G = 32 / BS;
  __shared__ int list[256];
  __shared__ int n_s;
  __shared__ VT red[8 * G * BS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane / BS, r = lane - g * BS;
  const int per = 256 / ch;
  if (threadIdx.x == 0) n_s = 0;
  __syncthreads();
  for (long long t0 = 0; (t0 * gridDim.x + blockIdx.x) * ch < mb; t0 += per) {
    const long long i =
        ((t0 + threadIdx.x / ch) * gridDim.x + blockIdx.x) * ch + threadIdx.x % ch;
    const bool hub = i < mb && __ldg(row + i + 1) - __ldg(row + i) > kLongSpmvRow;
    if (hub) list[atomicAdd(&n_s, 1)] = (int)i;
    if (!__syncthreads_or(hub)) continue;
    spmv_long_rows<BS, VT, XT, YT, VT, 8 * G>(list, n_s, row, col, val, x, y, y32, red, g < G,
                                              warp * G + g, r);
    if (threadIdx.x == 0) n_s = 0;
    __syncthreads();
  }
  dependency_wait();  // what follows in the stream comes after both kernels
}

// The same product with FP32 values for patterns with rows of more than
// kLongSpmvRow blocks (power-law: rows of ~7 blocks on average, many of one or
// two, hubs of up to 2000).  A group that walks a row alone waits for memory
// about once a batch, so the batches are deep; a warp owns `rw` consecutive
// rows and its lane groups take them one after another as they finish (the row
// pointers sit in the lanes' registers: taking a row is a ballot and two
// shuffles).  Rows of more than kLongSpmvRow blocks are summed by the CTA at
// the end.  Every sum runs in the order of a row per group.  62,500-row
// power-law ISAI factors, the apply: 8x8 blocks 151 -> 122 us, 4x4 92 -> 72 us.
constexpr int kUnevenMaxRows = 16;

template <int BS, class VT, class XT, class YT, class AccT, int U, int MINB>
__global__ void __launch_bounds__(256, MINB) k_bsr_spmv_uneven(int mb, int rw,
                                                               const int* __restrict__ row,
                                                               const int* __restrict__ col,
                                                               const VT* __restrict__ val,
                                                               const XT* __restrict__ x,
                                                               YT* __restrict__ y,
                                                               float* __restrict__ y32) {
  constexpr int G = 32 / BS;
  constexpr int NSLOT = 8 * kUnevenMaxRows;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ int long_slots[];  // [NSLOT] slots, then the partials
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane / BS, r = lane - g * BS;
  const long long r0 = ((long long)blockIdx.x * 8 + warp) * rw;
  const int nrow = (int)max(0ll, min((long long)rw, mb - r0));
  int sl = 0, el = 0;  // lane l < nrow: row r0 + l
  if (lane < nrow) {
    sl = __ldg(row + r0 + lane);
    el = __ldg(row + r0 + lane + 1);
  }
  const bool lng = el - sl > kLongSpmvRow;
  if (lane < kUnevenMaxRows) long_slots[warp * kUnevenMaxRows + lane] = lng ? (int)(r0 + lane) : -1;
  const unsigned skip = __ballot_sync(kAll, lng);
  if (lng) el = sl;
  int next = 0, cur = -1, p = 0, e = 0;
  AccT acc = 0;
  bool on = g < G;
  while (true) {
    const bool need = on && p >= e;
    if (need && cur >= 0 && !((skip >> cur) & 1u)) {
      y[(r0 + cur) * BS + r] = (YT)acc;
      if (y32) y32[(r0 + cur) * BS + r] = (float)acc;
    }
    const unsigned want = __ballot_sync(kAll, need && r == 0);
    const int idx = next + __popc(want & ((1u << (g * BS)) - 1u));
    next += __popc(want);
    const int from = min(idx, kUnevenMaxRows - 1);
    const int ps = __shfl_sync(kAll, sl, from), pe = __shfl_sync(kAll, el, from);
    if (need) {
      on = idx < nrow;
      cur = idx;
      p = ps;
      e = on ? pe : ps;
      acc = 0;
    }
    if (!__any_sync(kAll, on)) break;
    int c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = p + u < e ? __ldg(col + p + u) : -1;
    AccT a[U][BS];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c[u] >= 0) load_row<BS, VT, AccT>(val, p + u, r, a[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c[u] >= 0) {
        AccT xv[BS];
        load_x<BS, XT, AccT>(x, c[u], xv);
#pragma unroll
        for (int k = 0; k < BS; ++k) acc = fma(a[u][k], xv[k], acc);
      }
    p += U;
  }
  // one CTA barrier, which also says whether the CTA holds a long row
  if (__syncthreads_or(skip != 0))
    spmv_long_rows<BS, VT, XT, YT, AccT, 8 * G>(
        long_slots, NSLOT, row, col, val, x, y, y32, reinterpret_cast<AccT*>(long_slots + NSLOT),
        g < G, warp * G + g, r);
}

// The same product with FP64 values for those patterns, bound by the FP64 pipe
// (an FP64 warp instruction costs the same with one lane group active as with
// all, and a row per group left half of them idle; one SM alone takes 30 us for
// a hub of 1900 8x8 blocks).  A cluster of kBalCluster CTAs owns `rows`
// consecutive rows and splits their blocks, not their rows, evenly among all
// its lane groups: a group streams its run of blocks, storing a row's sum where
// the row ends inside the run.  A row that goes on into the next groups' runs is
// finished by the group it starts in, which adds the others' heads in order:
// those of its CTA from shared memory, one sum of each later CTA's (so a sum's
// order depends on the pattern alone).  62,500-row power-law ISAI factors, 8x8
// blocks (the apply: two products, 88 us of DFMA): 320 -> 152 us; 4x4 151 -> 69.
constexpr int kBalCluster = 8;
constexpr int kBalMaxRows = 1024;

template <int BS, int U, int MINB, bool TR>
__global__ void __launch_bounds__(256, MINB) k_bsr_spmv_balanced(
    int mb, int rows, const int* __restrict__ row, const int* __restrict__ col,
    const int* __restrict__ src, const double* __restrict__ val, const double* __restrict__ x,
    double* __restrict__ y, float* __restrict__ y32) {
  namespace cgr = cooperative_groups;
  constexpr int G = 32 / BS, NG = 8 * G, NGC = NG * kBalCluster;
  __shared__ int rp[kBalMaxRows + 1];
  __shared__ double head_s[NG][BS];
  __shared__ double chead_s[BS];
  cgr::cluster_group cl = cgr::this_cluster();
  const int rank = (int)cl.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane / BS, r = lane - g * BS;
  const long long r0 = (long long)(blockIdx.x / kBalCluster) * rows;
  const int n = (int)min((long long)rows, mb - r0);
  for (int t = threadIdx.x; t <= n; t += 256) rp[t] = __ldg(row + r0 + t);
  __syncthreads();
  for (int t = rank * 256 + threadIdx.x; t < n * BS; t += 256 * kBalCluster)
    if (rp[t / BS] == rp[t / BS + 1]) {  // empty rows
      y[r0 * BS + t] = 0.0;
      if (y32) y32[r0 * BS + t] = 0.f;
    }
  const int b0 = rp[0];
  const long long T = rp[n] - b0;
  auto start = [&](int q) { return b0 + (int)(T * q / NGC); };  // group q's run
  auto row_at = [&](int p) {  // last row starting at or before p: the one holding block p
    int lo = 0, up = n - 1;
    while (lo < up) {
      const int m = (lo + up + 1) >> 1;
      if (rp[m] <= p) lo = m; else up = m - 1;
    }
    return lo;
  };
  const int q0 = rank * NG, gi = q0 + warp * G + g;
  int p = g < G ? start(gi) : 0;
  const int hi = g < G ? start(gi + 1) : 0;
  double acc = 0.0;
  int cur = 0, e = 0;
  bool head = false, open = false;  // the row started before this run; acc is of a row
  if (p < hi) {
    cur = row_at(p);
    e = rp[cur + 1];
    head = rp[cur] < p;
    open = true;
  }
  while (p < hi) {
    int c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = p + u < hi ? __ldg(col + p + u) : -1;
    double a[U][BS];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c[u] >= 0) load_entry<BS, TR, double, double>(val, src, p + u, r, a[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c[u] >= 0) {
        double xv[BS];
        load_x<BS, double, double>(x, c[u], xv);
#pragma unroll
        for (int k = 0; k < BS; ++k) acc = fma(a[u][k], xv[k], acc);
        if (p + u + 1 == e) {  // the row ends here
          if (head) {
            head_s[gi - q0][r] = acc;
          } else {
            y[(r0 + cur) * BS + r] = acc;
            if (y32) y32[(r0 + cur) * BS + r] = (float)acc;
          }
          head = false;
          acc = 0.0;
          open = e < hi;
          if (open) {
            do e = rp[++cur + 1];
            while (e == p + u + 1);
          }
        }
      }
    p += U;
  }
  if (open && head) head_s[gi - q0][r] = acc;  // a row that fills the whole run
  __syncthreads();
  bool more = false;  // the row goes on in the next CTA
  if (open && !head) {
    for (int q = gi + 1; q < q0 + NG; ++q) {
      const int s = start(q);
      if (s >= e) break;
      if (s < start(q + 1)) acc += head_s[q - q0][r];
    }
    more = start(q0 + NG) < e;
    if (!more) {
      y[(r0 + cur) * BS + r] = acc;
      if (y32) y32[(r0 + cur) * BS + r] = (float)acc;
    }
  }
  // this CTA's part of a row that started in an earlier one
  const int cs = start(q0), ce = start(q0 + NG);
  if (threadIdx.x < BS && cs < ce) {
    const int k = row_at(cs), end = rp[k + 1];
    if (rp[k] < cs) {
      double t = 0.0;
      for (int q = q0; q < q0 + NG; ++q) {
        const int s = start(q);
        if (s >= end) break;
        if (s < start(q + 1)) t += head_s[q - q0][threadIdx.x];
      }
      chead_s[threadIdx.x] = t;
    }
  }
  cl.sync();
  if (more) {
    for (int c = rank + 1; c < kBalCluster; ++c) {
      const int s = start(c * NG);
      if (s >= e) break;
      if (s < start((c + 1) * NG)) acc += cl.map_shared_rank(chead_s, c)[r];
    }
    y[(r0 + cur) * BS + r] = acc;
    if (y32) y32[(r0 + cur) * BS + r] = (float)acc;
  }
  cl.sync();  // nobody leaves while its sums may be read
}

// Layout word of a matrix for the SpMV: bit 0 = rows of more than
// kLongSpmvRow blocks present; bit 1 = more than kWideSpmvRow blocks a row on
// average (FP32 values: one row per lane group).  The other bits, for the choice of
// the kernel alone (spmv_layout_word): the long rows hold few of the blocks and are
// not too long (FP64, FP32); all rows are about as long; few and wide rows.
constexpr int kLayoutLong = 1;
constexpr int kLayoutWide = 2;
constexpr int kLayoutHubs = 4;
constexpr int kLayoutHubs32 = 8;
constexpr int kLayoutAlike = 16;
constexpr int kLayoutFew = 32;
constexpr int kLayoutPublic = kLayoutLong | kLayoutWide;
constexpr int kWideSpmvRow = 5;

template <int BS, class VT, class XT, class YT>
int launch_spmv_hubs(int mb, const int* row, const int* col, const VT* val, const XT* x, YT* y,
                     cudaStream_t st, float* y32) {
  // a row a CTA and turn, then runs of up to a sector of row pointers
  constexpr int kCtas = 152 * 4;
  int ch = 1;
  while (ch < 8 && mb > ch * kCtas) ch *= 2;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min<unsigned>(ceil_div(mb, ch), kCtas));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  BILU_TRY_CUDA(cudaLaunchKernelEx(&cfg, k_spmv_hubs<BS, VT, XT, YT>, mb, ch, row, col, val, x, y,
                                   y32));
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

template <int BS, class VT, class XT, class YT, int RPG, int U, int MINB, bool TR = false>
int launch_spmv_cfg(int mb, const int* row, const int* col, const VT* val, const XT* x, YT* y,
                    cudaStream_t st, float* y32, bool dep, const int* src = nullptr,
                    bool hubs = false) {
  constexpr int G = 32 / BS;
  long long groups = (mb + RPG - 1) / RPG;
  long long warps = (groups + G - 1) / G;
  if constexpr (!TR) {
    if (hubs) {  // a chain of its own: the hubs' kernel reads x when this one has started
      k_bsr_spmv<BS, VT, XT, YT, VT, RPG, U, MINB, false, false, true>
          <<<ceil_div(warps, 8), 256, 0, st>>>(mb, row, col, src, val, x, y, y32);
      BILU_LAUNCH_CHECK();
      return launch_spmv_hubs<BS, VT, XT, YT>(mb, row, col, val, x, y, st, y32);
    }
  }
  // early starts follow a kernel that wrote x in the product's precision
  if constexpr (!TR && RPG == 1 && sizeof(XT) == sizeof(VT)) {
    if (dep) {
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[0].val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(ceil_div(warps, 8));
      cfg.blockDim = dim3(256);
      cfg.stream = st;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      BILU_TRY_CUDA(cudaLaunchKernelEx(&cfg, k_bsr_spmv<BS, VT, XT, YT, VT, RPG, U, MINB, TR, true, false>,
                                       mb, row, col, src, val, x, y, y32));
      BILU_LAUNCH_CHECK();
      return BILU_OK;
    }
  }
  k_bsr_spmv<BS, VT, XT, YT, VT, RPG, U, MINB, TR, false, false><<<ceil_div(warps, 8), 256, 0, st>>>(
      mb, row, col, src, val, x, y, y32);
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// Rows per warp: as many as leave two warps for every one that can be resident
// (balance), at least one per lane group, at most kUnevenMaxRows.
template <int BS, class XT, class YT, int U, int MINB>
int launch_spmv_uneven(int mb, const int* row, const int* col, const float* val, const XT* x,
                       YT* y, cudaStream_t st, float* y32) {
  const int rw = std::max(32 / BS, std::min(kUnevenMaxRows, mb / (152 * 8 * MINB * 2)));
  constexpr size_t smem = sizeof(int) * 8 * kUnevenMaxRows + sizeof(float) * 8 * (32 / BS) * BS;
  k_bsr_spmv_uneven<BS, float, XT, YT, float, U, MINB>
      <<<ceil_div(mb, 8ll * rw), 256, smem, st>>>(mb, rw, row, col, val, x, y, y32);
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// Rows per cluster: as many as leave one CTA (8x8 blocks: two) for every one that
// can be resident -- the two barriers of a cluster cost more than a second wave
// balances while the blocks are small (62,500 rows, the apply, 1 / 2 / 3 / 6
// waves: 4x4 69 / 77 / 92 / 141 us, 8x8 163 / 152 / 155 / 185 us) -- at least 64,
// at most kBalMaxRows.

template <int BS, int U, int MINB, bool TR>
int launch_spmv_balanced(int mb, const int* row, const int* col, const int* src,
                         const double* val, const double* x, double* y, cudaStream_t st,
                         float* y32) {
  const long long per = (long long)mb * kBalCluster / (152 * MINB * (BS == 8 ? 2 : 1));
  const int rows = (int)std::max(64ll, std::min((long long)kBalMaxRows, per));
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kBalCluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ceil_div(mb, rows) * kBalCluster);
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  BILU_TRY_CUDA(cudaLaunchKernelEx(&cfg, k_bsr_spmv_balanced<BS, U, MINB, TR>, mb, rows, row, col,
                                   src, val, x, y, y32));
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// The kernel and its configuration by the layout word; stencils and other patterns
// of short rows take k_bsr_spmv.
template <int BS, class VT, class XT, class YT>
int launch_spmv(int mb, const int* row, const int* col, const VT* val, const XT* x, YT* y,
                cudaStream_t st, int layout, float* y32, bool dep) {
  if (mb == 0) return BILU_OK;
  const bool hubs = (layout & (sizeof(VT) == 8 ? kLayoutHubs : kLayoutHubs32)) != 0;
  const int* none = nullptr;
  // Long rows that are neither few of the blocks nor like the others; in FP64 also
  // few wide rows, with or without long ones: a row a group leaves most of the
  // chip idle, or runs one FMA chain per row (4000 rows of 41 blocks, a row a group /
  // blocks split, us: 4x4 18.6 / 14.5, 8x8 41 / 33; 2000 of 201: 146 / 23, 187 / 62;
  // 16,000 of 41: 35 / 40, 92 / 95).  Where all rows are about as long and many, a
  // row a group it is (20,000 rows of 67: 4x4 64 / 70, 5x5 72 / 102, but 8x8
  // 189 / 181; FP32 21 / 94, 35 / 147, 64 / 159).
  if constexpr (sizeof(VT) == 8) {
    if ((layout & kLayoutFew) || ((layout & kLayoutLong) && !hubs &&
                                  !((layout & kLayoutAlike) && BS <= 5)))
      return launch_spmv_balanced<BS, 2, 4, false>(mb, row, col, nullptr, val, x, y, st, y32);
  } else if ((layout & kLayoutLong) && !hubs && !(layout & kLayoutAlike)) {
    return launch_spmv_uneven<BS, XT, YT, BS == 4 ? 4 : 8, BS == 4 ? 4 : 2>(mb, row, col, val, x, y,
                                                                           st, y32);
  }
  if constexpr (sizeof(VT) == 8) {
    return launch_spmv_cfg<BS, VT, XT, YT, 1, 1, BS <= 5 ? 6 : 5>(mb, row, col, val, x, y, st, y32,
                                                                  dep, none, hubs);
  } else if constexpr (BS == 8 && sizeof(XT) == 8) {
    // two rows of 8x8 blocks with FP64 x segments spill at 64 registers
    return launch_spmv_cfg<BS, VT, XT, YT, 1, 4, 4>(mb, row, col, val, x, y, st, y32, dep, none,
                                                    hubs);
  } else {
    // one row per group also where the first blocks are to wait in registers
    // for the launch before (two rows / one, the 512^2 5-point apply: bs 5 54.3
    // / 45.2 us, bs 8 80.4 / 68.9)
    if ((layout & kLayoutWide) || (BS != 4 && dep))
      return launch_spmv_cfg<BS, VT, XT, YT, 1, 4, 4>(mb, row, col, val, x, y, st, y32, dep, none,
                                                      hubs);
    // bs 4 rows of ~4 blocks (the ISAI triangles of a 7-point pattern): one
    // row per group at 32 registers, 8 CTAs per SM (0.2214 -> 0.2185 ms
    // for the 128^3 inner apply)
    if constexpr (BS == 4)
      return launch_spmv_cfg<BS, VT, XT, YT, 1, 4, 8>(mb, row, col, val, x, y, st, y32, dep, none,
                                                      hubs);
    return launch_spmv_cfg<BS, VT, XT, YT, 2, 4, 4>(mb, row, col, val, x, y, st, y32, dep, none,
                                                    hubs);
  }
}

// y = M^T x from M's values and the transposed pattern (launch_spmv's FP64
// kernels, so the sums run in the order of a product with the transposed
// matrix).
template <int BS>
int launch_spmv_t(int mb, const int* trow, const int* tcol, const int* src, const double* val,
                  const double* x, double* y, cudaStream_t st, int layout) {
  using D = double;
  if (layout & kLayoutLong)
    return launch_spmv_balanced<BS, 2, 4, true>(mb, trow, tcol, src, val, x, y, st, nullptr);
  if constexpr (BS <= 5)
    return launch_spmv_cfg<BS, D, D, D, 1, 1, 6, true>(mb, trow, tcol, val, x, y, st, nullptr,
                                                       false, src);
  else
    return launch_spmv_cfg<BS, D, D, D, 1, 1, 5, true>(mb, trow, tcol, val, x, y, st, nullptr,
                                                       false, src);
}

// Multi-RHS: Y[n,k] = M X[n,k], row-major with ld = k.  LPR lanes per block row
// (32 / LPR rows a warp), lane l owning right-hand sides l, l + LPR, ... (KW of
// them); every block is read by its lanes at once, row by row.  The FP64 product
// is bound by the FP64 pipe, whose warp instructions cost the same whatever the
// lanes, so LPR and KW are chosen to leave few of them without a right-hand
// side (launch_spmm).  With FP32 values X is rounded to FP32 where it is read
// and the sums are widened where they are stored, on the integer pipe: the
// conversion instructions run on the FP64 pipe and were the bound (512 x 512
// 5-point grid, 4x4 blocks, k 32: 342 -> 213 us, 92 us of HBM, bound by issue and
// L1).  Sums run in block order, then column order, whatever LPR and KW are (but
// for hub rows).
// With `hubs`, hub rows (spmm_hub: a group alone takes ~0.5 us a block, a
// millisecond for a hub of 2000) are left to k_spmm_hubs.
// vec: val starts on a 16-byte boundary (else blocks are read element by element)
template <int BS, class VT>
__device__ __forceinline__ void spmm_row(const VT* __restrict__ val, long long p, int r, int vec,
                                         VT* a) {
  if (vec) {
    load_row<BS, VT, VT>(val, p, r, a);
  } else {
#pragma unroll
    for (int kk = 0; kk < BS; ++kk) a[kk] = __ldg(val + (p * BS + r) * BS + kk);
  }
}

// X in the precision of the product
template <int N>
__device__ __forceinline__ void spmm_in(const double (&d)[N], double (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = d[i];
}
template <int N>
__device__ __forceinline__ void spmm_in(const double (&d)[N], float (&v)[N]) {
  if constexpr (N == 1) v[0] = narrow(d[0]);
  else narrow_all<N>(d, v);
}
// what a lane without a right-hand side works on (1: a zero would send its warp
// down narrow()'s branch)
constexpr double kNoRhs = 1.0;

template <class VT>
__device__ __forceinline__ double spmm_out(VT v) {
  if constexpr (sizeof(VT) == 4) return widen(v);
  else return v;
}

// A row that is summed apart: long, and much longer than the rows are on average.
// Where many rows are long a group per row fills the chip, and a CTA per row only
// adds barriers (20,000 rows of 67 4x4 blocks, FP32, k 32: 165 us with a group per
// row, 1845 with a CTA).  With few rows it does not: up to kHubFewRows every
// long row is a hub (a wave of CTAs; 300 rows of 300 8x8 blocks, FP64, k 1: 1455 us
// with a group per row, 50 so), and FP32 rows of twice that length up to 4096 rows
// (2000 rows of 201 8x8 blocks, k 1: 350 / 214).
constexpr int kHubFewRows = 152 * 4;
constexpr int kHubCtas = 2 * kHubFewRows;
template <class VT>
__device__ __forceinline__ bool spmm_hub(int len, int mb, const int* __restrict__ row) {
  if (len <= kLongSpmvRow) return false;
  if (mb <= kHubFewRows || (sizeof(VT) == 4 && mb <= 4096 && len > 2 * kLongSpmvRow)) return true;
  return (long long)len * mb > 4ll * (__ldg(row + mb) - __ldg(row));
}

// The hub rows of the product, a CTA each: its groups of LPR lanes share the row's
// blocks, U in flight each, and add their sums in a fixed order.  The CTAs look
// for hubs in turn, CH rows (a sector of row pointers on large matrices) at a
// time, so that neighbouring hubs go to different CTAs.  Started by programmatic
// dependent launch beside the other rows' kernel, whose rows of Y it does not
// touch, it ends after that one.  20,000-row power-law pattern, 4x4 blocks, k 32,
// the whole product, a warp per row / so: FP64 2507 / 530 us, FP32 1065 / 158.
template <int BS, class VT, int LPR>
__global__ void __launch_bounds__(256, BS <= 5 ? 3 : 2)
    k_spmm_hubs(int mb, int k, int vec, int ch, const int* __restrict__ row,
                const int* __restrict__ col, const VT* __restrict__ val,
                const double* __restrict__ X, double* __restrict__ Y) {
  constexpr int GW = 32 / LPR, NG = 8 * GW;
  constexpr int U = BS <= 5 ? 4 : 2;
  __shared__ VT part_s[8 * BS * LPR];
  __shared__ int list_s[256];
  const int lane = threadIdx.x & 31, l = lane & (LPR - 1), warp = threadIdx.x >> 5;
  const int gi = warp * GW + lane / LPR;
  const int per = 256 / ch;  // this CTA's turns looked through at once
  const int off = threadIdx.x % ch;
  for (long long t0 = 0; (t0 * gridDim.x + blockIdx.x) * ch < mb; t0 += per) {
    const long long i = ((t0 + threadIdx.x / ch) * gridDim.x + blockIdx.x) * ch + off;
    const bool hub = i < mb && spmm_hub<VT>(__ldg(row + i + 1) - __ldg(row + i), mb, row);
    if (!__syncthreads_or(hub)) continue;
    list_s[threadIdx.x] = hub ? (int)i : -1;
    __syncthreads();
    unsigned todo = 0;  // of the list's next 32 entries, the same in every warp
    for (int h = 0; h < 256 || todo;) {
      if (!todo) {
        todo = __ballot_sync(0xffffffffu, list_s[h + lane] >= 0);
        h += 32;
        continue;
      }
      const int br = list_s[h - 33 + __ffs(todo)];
      todo &= todo - 1;
      const int hs = __ldg(row + br), he = __ldg(row + br + 1);
      for (int k0 = 0; k0 < k; k0 += LPR) {
        const bool in = k0 + l < k;
        const double* Xc = X + k0 + l;
        VT acc[BS];
#pragma unroll
        for (int r = 0; r < BS; ++r) acc[r] = 0;
        for (int q = hs + gi; q < he; q += NG * U) {
          double xd[U][BS];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const double* xb = Xc + (long long)__ldg(col + min(q + u * NG, he - 1)) * BS * k;
#pragma unroll
            for (int kk = 0; kk < BS; ++kk)
              xd[u][kk] = in ? __ldg(xb + (long long)kk * k) : kNoRhs;
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (q + u * NG >= he) break;
            VT xv[BS];
            spmm_in<BS>(xd[u], xv);
#pragma unroll
            for (int r = 0; r < BS; ++r) {
              VT a[BS];
              spmm_row<BS, VT>(val, q + u * NG, r, vec, a);
#pragma unroll
              for (int kk = 0; kk < BS; ++kk) acc[r] = fma(a[kk], xv[kk], acc[r]);
            }
          }
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < BS; ++r) {
#pragma unroll
          for (int o = LPR; o < 32; o <<= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
          if (lane < LPR) part_s[(warp * BS + r) * LPR + l] = acc[r];
        }
        __syncthreads();
        for (int t = threadIdx.x; t < BS * LPR; t += 256) {
          const int r = t / LPR, c = k0 + t % LPR;
          VT sum = 0;
#pragma unroll
          for (int w = 0; w < 8; ++w) sum += part_s[(w * BS + r) * LPR + t % LPR];
          if (c < k) Y[((long long)br * BS + r) * k + c] = spmm_out(sum);
        }
        __syncthreads();
      }
    }
    __syncthreads();  // the list is written again
  }
  dependency_wait();  // what follows in the stream comes after both kernels
}

// FULL: k is LPR KW and val is aligned, known to the compiler (immediate offsets,
// no predicates or branches).
// (8x8 blocks, FP64: 6 CTAs per SM, not the 4 of 56 registers: 5000 rows of 41
// blocks, k 32, 1023 -> 890 us.)
template <int BS, class VT, int LPR, int KW, bool FULL>
__global__ void __launch_bounds__(256, sizeof(VT) == 8 && BS == 8 && KW == 1 && FULL ? 6 : 0)
    k_bsr_spmm(int mb, int k_any, int vec_any, int hubs, const int* __restrict__ row,
               const int* __restrict__ col, const VT* __restrict__ val,
               const double* __restrict__ X, double* __restrict__ Y) {
  dependents_launch();  // k_spmm_hubs
  const int k = FULL ? LPR * KW : k_any, vec = FULL ? 1 : vec_any;
  const int lane = threadIdx.x & 31, l = lane & (LPR - 1);
  const long long br =
      ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 / LPR) + lane / LPR;
  if (br >= mb) return;
  const int e = __ldg(row + br + 1);
  int p = __ldg(row + br);
  if (hubs && spmm_hub<VT>(e - p, mb, row)) return;
  VT acc[KW][BS];
#pragma unroll
  for (int w = 0; w < KW; ++w)
#pragma unroll
    for (int r = 0; r < BS; ++r) acc[w][r] = 0;
  int bc = p < e ? __ldg(col + p) : 0;
  for (; p < e; ++p) {
    const double* xb = X + (long long)bc * BS * k + l;
    double xd[BS * KW];
#pragma unroll
    for (int kk = 0; kk < BS; ++kk)
#pragma unroll
      for (int w = 0; w < KW; ++w)
        xd[kk * KW + w] = l + LPR * w < k ? __ldg(xb + kk * k + LPR * w) : kNoRhs;
    if (p + 1 < e) bc = __ldg(col + p + 1);
    // FP32: the next block's X and values on their way (the grid above 250 -> 213 us;
    // 2000 rows of 67 blocks, where every block waited for its values, 50 -> 41; the
    // FP64 product has the time)
    if (sizeof(VT) == 4 && p + 1 < e)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(X + (long long)bc * BS * k + l));
    {
      constexpr int LW = 128 / (int)sizeof(VT);  // a line a lane, and the block's last element
      if (sizeof(VT) == 4 && p + 1 < e && (l - 1) * LW < BS * BS)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(val + (long long)(p + 1) * BS * BS +
                                                      min(l * LW, BS * BS - 1)));
    }
    VT xv[BS * KW];
#pragma unroll
    for (int i = 0; i < BS * KW; ++i) spmm_in<1>({xd[i]}, reinterpret_cast<VT(&)[1]>(xv[i]));
#pragma unroll
    for (int r = 0; r < BS; ++r) {
      VT a[BS];
      spmm_row<BS, VT>(val, p, r, vec, a);
#pragma unroll
      for (int kk = 0; kk < BS; ++kk)
#pragma unroll
        for (int w = 0; w < KW; ++w) acc[w][r] = fma(a[kk], xv[kk * KW + w], acc[w][r]);
    }
  }
#pragma unroll
  for (int w = 0; w < KW; ++w)
    if (l + LPR * w < k)
#pragma unroll
      for (int r = 0; r < BS; ++r) Y[(br * BS + r) * k + l + LPR * w] = spmm_out(acc[w][r]);
}

template <int BS, class VT, int LPR, int KW>
int launch_spmm_cfg(int mb, int k, const int* row, const int* col, const VT* val, const double* X,
                    double* Y, cudaStream_t st) {
  const int vec = (uintptr_t)val % 16 == 0;
  const unsigned grid = ceil_div(mb, 8 * (32 / LPR));
  // A few rows are not worth a second launch for the long ones among them: a
  // square matrix without repeated columns has none there, and a slice of a
  // wider one keeps a group per row whatever its rows hold.
  const int hubs = mb > kLongSpmvRow;
  if (k == LPR * KW && vec)
    k_bsr_spmm<BS, VT, LPR, KW, true><<<grid, 256, 0, st>>>(mb, k, vec, hubs, row, col, val, X, Y);
  else
    k_bsr_spmm<BS, VT, LPR, KW, false><<<grid, 256, 0, st>>>(mb, k, vec, hubs, row, col, val, X, Y);
  BILU_LAUNCH_CHECK();
  if (!hubs) return BILU_OK;
  // a row a CTA and turn up to kHubCtas, then runs of up to a sector of row
  // pointers
  int ch = 1;
  while (ch < 8 && mb > ch * kHubCtas) ch *= 2;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min<unsigned>(ceil_div(mb, ch), kHubCtas));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  BILU_TRY_CUDA(cudaLaunchKernelEx(&cfg, k_spmm_hubs<BS, VT, LPR>, mb, k, vec, ch, row, col, val,
                                   X, Y));
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// The lanes' padding decides: k right-hand sides take ceil(k / LPR) LPR slots.
template <int BS, class VT>
int launch_spmm(int mb, int k, const int* row, const int* col, const VT* val, const double* X,
                double* Y, cudaStream_t st) {
  if (mb == 0) return BILU_OK;
  if (k <= 4) return launch_spmm_cfg<BS, VT, 4, 1>(mb, k, row, col, val, X, Y, st);
  if (k <= 8) return launch_spmm_cfg<BS, VT, 8, 1>(mb, k, row, col, val, X, Y, st);
  if (k <= 16) return launch_spmm_cfg<BS, VT, 16, 1>(mb, k, row, col, val, X, Y, st);
  if (k <= 24) return launch_spmm_cfg<BS, VT, 8, 3>(mb, k, row, col, val, X, Y, st);
  if (k <= 32) return launch_spmm_cfg<BS, VT, 32, 1>(mb, k, row, col, val, X, Y, st);
  if (k <= 48) return launch_spmm_cfg<BS, VT, 16, 3>(mb, k, row, col, val, X, Y, st);
  return launch_spmm_cfg<BS, VT, 32, 2>(mb, k, row, col, val, X, Y, st);
}

// d32 = s rounded to FP32, d0 and d1 (optional) copies of s.  Bound by HBM: four
// elements a thread in 16-byte accesses, rounded on the integer pipe (the
// conversion instruction runs on the FP64 pipe, 14 us for 8.4 M elements
// beside 15 of HBM).  vec: every pointer is on a 16-byte boundary.
__global__ void __launch_bounds__(256) k_copy_values(size_t n, int vec,
                                                     const double* __restrict__ s,
                                                     double* __restrict__ d0,
                                                     double* __restrict__ d1,
                                                     float* __restrict__ d32) {
  dependents_launch();
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t n4 = vec ? n / 4 : 0;
  for (size_t i = t; i < n4; i += stride) {
    const double2 a = ld_stream(reinterpret_cast<const double2*>(s) + 2 * i),
                  b = ld_stream(reinterpret_cast<const double2*>(s) + 2 * i + 1);
    if (d0) {
      reinterpret_cast<double2*>(d0)[2 * i] = a;
      reinterpret_cast<double2*>(d0)[2 * i + 1] = b;
    }
    if (d1) {
      reinterpret_cast<double2*>(d1)[2 * i] = a;
      reinterpret_cast<double2*>(d1)[2 * i + 1] = b;
    }
    if (d32) {
      const double v[4] = {a.x, a.y, b.x, b.y};
      float f[4];
      narrow_all<4>(v, f);
      reinterpret_cast<float4*>(d32)[i] = make_float4(f[0], f[1], f[2], f[3]);
    }
  }
  for (size_t i = 4 * n4 + t; i < n; i += stride) {
    const double v = s[i];
    if (d0) d0[i] = v;
    if (d1) d1[i] = v;
    if (d32) d32[i] = narrow(v);
  }
}

template <int BS>
int spmv_f64(int mb, const int* row, const int* col, const double* val, const double* x,
             double* y, cudaStream_t st, int lr, bool dep) {
  return launch_spmv<BS, double, double, double>(mb, row, col, val, x, y, st, lr, nullptr, dep);
}

template <int BS>
int spmv_f32(int mb, const int* row, const int* col, const float* val, const void* x, int x32,
             void* y, int y32, cudaStream_t st, int lr, bool dep) {
  if (x32 && y32)
    return launch_spmv<BS, float, float, float>(mb, row, col, val, (const float*)x, (float*)y, st,
                                                lr, nullptr, dep);
  if (x32)
    return launch_spmv<BS, float, float, double>(mb, row, col, val, (const float*)x, (double*)y,
                                                 st, lr, nullptr, dep);
  if (y32)
    return launch_spmv<BS, float, double, float>(mb, row, col, val, (const double*)x, (float*)y,
                                                 st, lr, nullptr, dep);
  return launch_spmv<BS, float, double, double>(mb, row, col, val, (const double*)x, (double*)y,
                                                st, lr, nullptr, dep);
}

// FP32 values and x, FP64 y plus its FP32 copy y32
template <int BS>
int spmv_f32_dual(int mb, const int* row, const int* col, const float* val, const float* x,
                  double* y, float* y32, cudaStream_t st, int lr, bool dep) {
  return launch_spmv<BS, float, float, double>(mb, row, col, val, x, y, st, lr, y32, dep);
}

// out[0] = the longest row, out[1] = the blocks in long rows
__global__ void k_row_len_max(int mb, const int* __restrict__ row, int* out) {
  int m = 0, h = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < mb;
       i += (long long)gridDim.x * blockDim.x) {
    const int n = __ldg(row + i + 1) - __ldg(row + i);
    m = max(m, n);
    if (n > kLongSpmvRow) h += n;
  }
  m = __reduce_max_sync(0xffffffffu, m);
  h = __reduce_add_sync(0xffffffffu, h);
  if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(out, m);
  if ((threadIdx.x & 31) == 0 && h > 0) atomicAdd(out + 1, h);
}

template <int BS>
int spmm_f64(int mb, int k, const int* row, const int* col, const double* val, const double* X,
             double* Y, cudaStream_t st) {
  return launch_spmm<BS, double>(mb, k, row, col, val, X, Y, st);
}
template <int BS>
int spmm_f32(int mb, int k, const int* row, const int* col, const float* val, const double* X,
             double* Y, cudaStream_t st) {
  return launch_spmm<BS, float>(mb, k, row, col, val, X, Y, st);
}

}  // namespace

// The layout word of a pattern of mb rows and nnzb blocks, its longest row and the
// blocks in long rows given.  Long rows go apart (k_spmv_hubs) up to a length that
// one SM gets through while the others do the rest, and to a share of the blocks
// from which a split of all blocks is the better balance.  40^3 grids, rows apart /
// balanced (FP64) or uneven (FP32), us, 4x4 and 8x8 --
// FP64: 50 rows of 200 (2%) 23 / 32, 62 / 72; 1000 of 100 (16%) 42 / 37, 92 / 82;
// 20 of 1000 (4%) 39 / 31, 106 / 71;
// FP32: 50 of 200 9.5 / 12.4, 26 / 35; 1000 of 100 12.6 / 20.5, 37 / 45; 20 of 1000
// 14.5 / 14.5, 46 / 36.
// Hubs of 1000 are worth it again on 80^3 (5x5, FP32, 90 / 97), and a few hubs on
// any small pattern (700 rows, 3 of 80, 4x4, FP64, 8.3 / 12.3).
int spmv_layout_word(int mb, long long nnzb, int longest, long long hubs) {
  int w = 0;
  if (nnzb > (long long)kWideSpmvRow * mb) w |= kLayoutWide;
  if ((long long)longest * mb <= 2 * nnzb) w |= kLayoutAlike;
  if ((mb <= 8192 && nnzb >= 32ll * mb) || (mb <= 4096 && nnzb >= 24ll * mb)) w |= kLayoutFew;
  if (longest > kLongSpmvRow) {
    w |= kLayoutLong;
    const bool fits = 2000ll * longest < nnzb;
    if (!(w & kLayoutAlike)) {
      if ((fits || longest <= 4 * kLongSpmvRow) && (10 * hubs < nnzb || hubs <= 4096))
        w |= kLayoutHubs;
      if ((fits || longest <= 8 * kLongSpmvRow) && (2 * hubs < nnzb || hubs <= 4096))
        w |= kLayoutHubs32;
    }
  }
  return w;
}

// SpMV layout word of a block pattern (see kLayoutLong): one reduction
// over the row pointers into d_words (two device ints), then a synchronising
// read of it and of the block count row[mb].  The engine calls it once per
// matrix at setup.
int spmv_layout_of(int mb, int bs, const int* row, void* d_words, cudaStream_t st,
                   int* h_layout) {
  (void)bs;
  *h_layout = 0;
  if (mb <= 0) return BILU_OK;
  int h[3] = {0, 0, 0};  // longest row, blocks in long rows, blocks
  int* d = static_cast<int*>(d_words);
  BILU_TRY_CUDA(cudaMemsetAsync(d, 0, sizeof(int) * 2, st));
  k_row_len_max<<<(unsigned)std::min<long long>(ceil_div(mb, 256), 152 * 8), 256, 0, st>>>(
      mb, row, d);
  BILU_LAUNCH_CHECK();
  BILU_TRY_CUDA(cudaMemcpyAsync(&h[0], d, sizeof(int) * 2, cudaMemcpyDeviceToHost, st));
  BILU_TRY_CUDA(cudaMemcpyAsync(&h[2], row + mb, sizeof(int), cudaMemcpyDeviceToHost, st));
  BILU_TRY_CUDA(cudaStreamSynchronize(st));
  *h_layout = spmv_layout_word(mb, h[2], h[0], h[1]);
  return BILU_OK;
}

namespace {

__device__ int g_layout_word[2];  // scratch of the cached check (under its lock)

// The standalone entry points do not know the pattern: the answer is cached
// per (row pointer array, block rows, block size), most recent first.  A
// stale entry (a buffer reused for another pattern) can only cost speed:
// every kernel is exact for any row length.
struct LayoutEntry {
  const int* row;
  int mb, bs, layout;
};
std::mutex g_layout_mu;
LayoutEntry g_layout_cache[16] = {};
int g_layout_next = 0;

// under g_layout_mu: the entry of (row, mb, bs), or null
LayoutEntry* layout_find(int mb, int bs, const int* row) {
  for (LayoutEntry& e : g_layout_cache)
    if (e.row == row && e.mb == mb && e.bs == bs && row) return &e;
  return nullptr;
}

int layout_cached(int mb, int bs, const int* row, cudaStream_t st, int* out) {
  std::lock_guard<std::mutex> lock(g_layout_mu);
  if (const LayoutEntry* e = layout_find(mb, bs, row)) {
    *out = e->layout;
    return BILU_OK;
  }
  void* words = nullptr;
  BILU_TRY_CUDA(cudaGetSymbolAddress(&words, g_layout_word));
  int layout = 0;
  BILU_TRY(spmv_layout_of(mb, bs, row, words, st, &layout));
  g_layout_cache[g_layout_next] = LayoutEntry{row, mb, bs, layout};
  g_layout_next = (g_layout_next + 1) % 16;
  *out = layout;
  return BILU_OK;
}

}  // namespace

// internal entry point used by the solver; layout: the pattern's layout
// word when the caller knows it (spmv_layout_of), -1 to look it up
int spmv_any(int mb, int bs, int prec, const int* row, const int* col, const void* val,
             const void* x, int x32, void* y, int y32, cudaStream_t st, int layout, bool dep) {
  int lr = layout;
  if (layout < 0) BILU_TRY(layout_cached(mb, bs, row, st, &lr));
  if (prec == BILU_FP64) {
    if (x32 || y32) return BILU_ERR_ARG;
    return BILU_DISPATCH_BS(bs, spmv_f64, mb, row, col, (const double*)val, (const double*)x,
                            (double*)y, st, lr, dep);
  }
  return BILU_DISPATCH_BS(bs, spmv_f32, mb, row, col, (const float*)val, x, x32, y, y32, st, lr,
                          dep);
}

// y = M^T x: trow / tcol the transposed pattern, src the block of M each of its
// entries stands for, longest its longest row.
int spmv_gather_t(int mb, int bs, const int* trow, const int* tcol, const int* src,
                  const double* val, const double* x, double* y, int longest,
                  cudaStream_t st) {
  const int layout = longest > kLongSpmvRow ? kLayoutLong : 0;
  return BILU_DISPATCH_BS(bs, launch_spmv_t, mb, trow, tcol, src, val, x, y, st, layout);
}

int copy_values(size_t count, const double* src, double* d0, double* d1, float* d32,
                cudaStream_t st) {
  if (count == 0) return BILU_OK;
  const int vec = ((uintptr_t)src | (uintptr_t)d0 | (uintptr_t)d1 | (uintptr_t)d32) % 16 == 0;
  const size_t threads = vec ? (count + 3) / 4 : count;
  k_copy_values<<<(unsigned)std::min<size_t>((threads + 255) / 256, 152 * 16), 256, 0, st>>>(
      count, vec, src, d0, d1, d32);
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// FP32 path: b is rounded to FP32 once (n conversions; converting inside the
// SpMV would cost one FP64-pipe conversion per block element, the slowest
// operation on GB300), staged in the output buffer (n doubles hold n floats),
// then y32 = M_L b32 and x = M_U y32 with FP32 accumulation.
int isai_apply_impl(int nb, int bs, int prec, const int* Lrow, const int* Lcol, const void* Lval,
                    const int* Urow, const int* Ucol, const void* Uval, const double* b,
                    void* tmp, double* x, cudaStream_t st, int longL, int longU) {
  if (prec == BILU_FP32) {
    float* b32 = reinterpret_cast<float*>(x);
    BILU_TRY(copy_values((size_t)nb * bs, b, nullptr, nullptr, b32, st));
    BILU_TRY(spmv_any(nb, bs, prec, Lrow, Lcol, Lval, b32, 1, tmp, 1, st, longL, true));
    return spmv_any(nb, bs, prec, Urow, Ucol, Uval, tmp, 1, x, 0, st, longU, true);
  }
  BILU_TRY(spmv_any(nb, bs, prec, Lrow, Lcol, Lval, b, 0, tmp, 0, st, longL, false));
  return spmv_any(nb, bs, prec, Urow, Ucol, Uval, tmp, 0, x, 0, st, longU, true);
}

// Solver form: the FP32 copy of the input is already there (written by the
// kernel that produced the FP64 basis vector).
int isai_apply_f32_staged(int nb, int bs, const int* Lrow, const int* Lcol, const float* Lval,
                          const int* Urow, const int* Ucol, const float* Uval, const float* b32,
                          float* tmp, double* x, cudaStream_t st, float* x32, int longL,
                          int longU) {
  BILU_TRY(spmv_any(nb, bs, BILU_FP32, Lrow, Lcol, Lval, b32, 1, tmp, 1, st, longL, false));
  if (x32) {  // x also in FP32 (input of an FP32 operator product)
    int lr = longU;
    if (longU < 0) BILU_TRY(layout_cached(nb, bs, Urow, st, &lr));
    return BILU_DISPATCH_BS(bs, spmv_f32_dual, nb, Urow, Ucol, Uval, tmp, x, x32, st, lr,
                            true);
  }
  return spmv_any(nb, bs, BILU_FP32, Urow, Ucol, Uval, tmp, 1, x, 0, st, longU, true);
}

}  // namespace bilu

using namespace bilu;

extern "C" int bilu_bcsr_spmv(int mb, int bs, const int* d_row, const int* d_col,
                              const double* d_val, const double* d_x, double* d_y,
                              bilu_stream_t stream) {
  if (mb < 0 || (mb > 0 && (!d_row || !d_col || !d_val || !d_x || !d_y))) return BILU_ERR_ARG;
  if (!bs_supported(bs)) return BILU_ERR_UNSUPPORTED;
  return spmv_any(mb, bs, BILU_FP64, d_row, d_col, d_val, d_x, 0, d_y, 0, S(stream), -1, false);
}

extern "C" int bilu_spmv_layout(int mb, int bs, const int* d_row, bilu_stream_t stream,
                                int* h_layout) {
  if (mb < 0 || !h_layout || (mb > 0 && !d_row)) return BILU_ERR_ARG;
  if (!bs_supported(bs)) return BILU_ERR_UNSUPPORTED;
  BILU_TRY(layout_cached(mb, bs, d_row, S(stream), h_layout));
  *h_layout &= kLayoutPublic;
  return BILU_OK;
}

extern "C" int bilu_debug_spmv_layout_set(int mb, int bs, const int* d_row, int layout) {
  if (mb < 0 || (mb > 0 && !d_row) || layout < 0 || layout > kLayoutPublic)
    return BILU_ERR_ARG;
  if (!bs_supported(bs)) return BILU_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_layout_mu);
  if (LayoutEntry* e = layout_find(mb, bs, d_row)) {
    e->layout = layout;
  } else {
    g_layout_cache[g_layout_next] = LayoutEntry{d_row, mb, bs, layout};
    g_layout_next = (g_layout_next + 1) % 16;
  }
  return BILU_OK;
}

extern "C" int bilu_bcsr_spmv_f32(int mb, int bs, const int* d_row, const int* d_col,
                                  const float* d_val, const void* d_x, int x_fp32, void* d_y,
                                  int y_fp32, bilu_stream_t stream) {
  if (mb < 0 || (mb > 0 && (!d_row || !d_col || !d_val || !d_x || !d_y))) return BILU_ERR_ARG;
  if (!bs_supported(bs)) return BILU_ERR_UNSUPPORTED;
  return spmv_any(mb, bs, BILU_FP32, d_row, d_col, d_val, d_x, x_fp32 != 0, d_y, y_fp32 != 0,
                  S(stream), -1, false);
}

extern "C" int bilu_bcsr_spmm(int mb, int bs, int k, const int* d_row, const int* d_col,
                              const double* d_val, const double* d_X, double* d_Y,
                              bilu_stream_t stream) {
  if (mb < 0 || k < 1 || k > 64) return BILU_ERR_ARG;
  if (!bs_supported(bs)) return BILU_ERR_UNSUPPORTED;
  return BILU_DISPATCH_BS(bs, spmm_f64, mb, k, d_row, d_col, d_val, d_X, d_Y, S(stream));
}

extern "C" int bilu_bcsr_spmm_f32(int mb, int bs, int k, const int* d_row, const int* d_col,
                                  const float* d_val, const double* d_X, double* d_Y,
                                  bilu_stream_t stream) {
  if (mb < 0 || k < 1 || k > 64) return BILU_ERR_ARG;
  if (!bs_supported(bs)) return BILU_ERR_UNSUPPORTED;
  return BILU_DISPATCH_BS(bs, spmm_f32, mb, k, d_row, d_col, d_val, d_X, d_Y, S(stream));
}

extern "C" int bilu_convert_f64_to_f32(size_t count, const double* d_src, float* d_dst,
                                       bilu_stream_t stream) {
  if (count == 0) return BILU_OK;
  if (!d_src || !d_dst) return BILU_ERR_ARG;
  return copy_values(count, d_src, nullptr, nullptr, d_dst, S(stream));
}

extern "C" int bilu_isai_apply(int nb, int bs, int prec, const int* d_Lrow, const int* d_Lcol,
                               const void* d_Lval, const int* d_Urow, const int* d_Ucol,
                               const void* d_Uval, const double* d_b, void* d_tmp, double* d_x,
                               bilu_stream_t stream) {
  if (nb < 0 || (prec != BILU_FP64 && prec != BILU_FP32)) return BILU_ERR_ARG;
  if (!bs_supported(bs)) return BILU_ERR_UNSUPPORTED;
  return isai_apply_impl(nb, bs, prec, d_Lrow, d_Lcol, d_Lval, d_Urow, d_Ucol, d_Uval, d_b,
                         d_tmp, d_x, S(stream), -1, -1);
}
